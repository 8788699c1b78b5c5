"""List rebuild where its paths change: columns above one sort's size, pieces
with more hits than shared memory keeps, more masks than jobs, atoms outside
the box by more than the stored image shift, and undersized capacities; every
list bit for bit that of the CPU restatement."""
import dataclasses

import numpy as np
import pytest
import torch

import oracle
from blade_b200 import systems
from blade_b200.nbdirect import NbDirect

pytestmark = pytest.mark.gpu

KEYS = ("wrap", "blockBounds", "sortedAtom", "slotAtom", "bmin", "bmax", "candStart", "cand", "candExcl", "masks")


def _water(n, spacing=18.856 / 6, **kw):
    """n[0] x n[1] x n[2] lattice waters."""
    g = np.stack(np.meshgrid(*[(np.arange(k) + 0.5) * spacing for k in n], indexing="ij"), -1).reshape(-1, 3)
    s = systems.water_box(3, 6)
    rng = np.random.default_rng(3)
    xyz = systems.place_waters(rng, g, 0.3).astype(np.float32)
    nb = np.tile(s.nbonds[:3], len(g))
    return dataclasses.replace(s, xyz=xyz, nbonds=nb, excl=systems.water_excl(0, len(g)),
                               box=np.float32([k * spacing for k in n]), **kw)


def _compare(s):
    nb = NbDirect(s)
    pos = nb.positions_tensor()
    for _ in range(2):                                    # a second build of the same list
        nb.update_domdec(pos, True)
        g, o = nb.get_list(), oracle.build_list(s)
        for k in KEYS:
            assert np.array_equal(g[k], o[k]), k
    assert nb.list_sizes()["tiles"] == len(o["cand"])
    nb.close()


def test_tall_columns(cuda):
    _compare(_water((6, 6, 60)))                          # ~700 atoms a column: bitonic sort
    _compare(_water((6, 6, 500)))                         # ~6,000: counted in global memory


def test_many_hits_and_masks(cuda):
    s = _water((10, 9, 8), rCut=12.0, rSwitch=10.0, cullPad=8.0)
    _compare(s)                                           # several images of a block, many hits a piece
    rng = np.random.default_rng(5)
    a = rng.integers(0, 32, 60)                           # partners all over: mask words of many blocks
    extra = np.stack([a, rng.integers(0, s.N, 60)], 1)
    extra = extra[extra[:, 0] != extra[:, 1]]
    _compare(dataclasses.replace(s, excl=np.concatenate([s.excl, extra, extra[:, ::-1]]).astype(np.int32)))


def test_unwrapped_and_far_atoms(cuda):
    s = _water((7, 7, 7))
    x = s.xyz.reshape(-1, 3, 3).copy()
    x[::3] += 5 * s.box                                   # whole molecules some boxes away
    x[1::7] -= 3 * s.box
    _compare(dataclasses.replace(s, xyz=x.reshape(-1, 3)))
    far = s.xyz.copy()
    far[30:33] += np.float32(200) * s.box                 # beyond the 127 images of the stored shift
    _compare(dataclasses.replace(s, xyz=far))


@pytest.mark.parametrize("tiles,masks,work", [(16, 2, 4), (100000, 2, 4), (100000, 100000, 3), (20, 100000, 100000)])
def test_capacities_regrow_to_the_same_list(cuda, tiles, masks, work):
    s = systems.msld_water(9)
    nb = NbDirect(s)
    nb.reserve(tiles=tiles, masks=masks, work=work)
    pos = nb.positions_tensor()
    nb.update_domdec(pos, True)
    assert nb.status() & 15 == 0
    g, o = nb.get_list(), oracle.build_list(s)
    for k in KEYS:
        assert np.array_equal(g[k], o[k]), k
    sz = nb.list_sizes()
    assert sz["tiles"] == len(o["cand"]) and sz["masks"] == len(o["masks"])
    nb.close()


def test_tail_items_and_order_do_not_change_the_sums(cuda):
    """Work items with and without a tail, in list order and measured order."""
    s = systems.water_box(6, n_side=10, box=31.43, rCut=12.0, rSwitch=10.0, beta=0.32)
    ref = oracle.nbdirect(s)["grad"]
    for tiles, tail in ((8, 0), (8, 2), (16, 8), (1, 0)):
        nb = NbDirect(s)
        nb.set_tuning(tiles, tail_items=tail)
        pos = nb.positions_tensor()
        nb.update_domdec(pos, True)
        f = [nb.evaluate(pos)[0] for _ in range(3)]       # the second and third follow the measured order
        assert torch.equal(f[0], f[1]) and torch.equal(f[0], f[2])
        g = f[0].cpu().numpy()
        assert np.sqrt(((g - ref) ** 2).sum()) <= 1e-5 * np.sqrt((ref ** 2).sum())
        nb.close()
