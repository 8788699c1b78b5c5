"""Pair-kernel rounds at the sizes where they are padded or one half of a block
is empty, and the default split of the work list."""
import dataclasses

import numpy as np
import pytest
import torch

import oracle
from blade_b200 import systems
from blade_b200.nbdirect import NbDirect

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _first(s, n):
    """The first n atoms of a system."""
    return dataclasses.replace(s, xyz=s.xyz[:n].copy(), nbonds=s.nbonds[:n].copy(), excl=s.excl[(s.excl < n).all(1)],
                               bonds=None, bond_param=None)


def _check(s, **tuning):
    nb = NbDirect(s)
    if tuning:
        nb.set_tuning(**tuning)
    pos = nb.positions_tensor()
    nb.update_domdec(pos, True)
    nb.set_counting(True)
    lam = nb.lambdas_tensor()
    f, l, e = nb.evaluate(pos, lam)
    o = oracle.nbdirect(s, lam=lam.cpu().numpy().astype(np.float64))
    assert nb.status() == 0
    # a pair whose FP32 distance rounds across the cutoff may be counted on either side
    assert abs(nb.pair_count() - o["pairs"]) <= 2
    g = f.cpu().numpy()
    assert np.sqrt(((g - o["grad"]) ** 2).sum()) <= TOL * max(np.sqrt((o["grad"] ** 2).sum()), 1e-3)
    assert abs(float(e[0]) - o["energy"]) <= TOL * max(abs(o["energy"]), s.N)
    lo = np.asarray(o["lambdaForce"])
    assert np.abs(l.cpu().numpy()[1:] - lo[1:]).max(initial=0.0) <= TOL * max(np.abs(lo).max(initial=0.0), s.N)
    # the force-only kernel gives the forces of the energy kernel to rounding
    f2, _, _ = nb.evaluate(pos, lam, calc_energy=False)
    assert float((f2 - f).norm()) <= TOL * max(float(f.norm()), 1e-3)
    nb.close()


# one atom, a half block, a half and one, a whole block and one, whole blocks
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 31, 32, 33, 48, 65, 95, 96, 97, 200])
@pytest.mark.parametrize("methods", [(1, 0), (0, 0), (2, 2)])
def test_partial_blocks(cuda, n, methods):
    s = _first(systems.water_box(4), n)
    s.elecMethod, s.vdwMethod = methods
    _check(s)


@pytest.mark.parametrize("n", [9, 33, 64, 100, 131, 200])
@pytest.mark.parametrize("soft", [True, False])
def test_partial_msld_blocks(cuda, n, soft):
    s = _first(systems.msld_water(11), n)
    s.msld = dataclasses.replace(s.msld, useSoftCore=soft)
    _check(s)


@pytest.mark.parametrize("tiles,tail", [(1, 0), (2, 2), (8, 0), (32, 0)])
def test_rounds_over_item_sizes(cuda, tiles, tail):
    _check(systems.msld_water(12), tiles_per_work=tiles, tail_items=tail)


def test_default_split_follows_the_replica_and_keeps_the_list(cuda):
    small, large = systems.water_box(5), systems.water_box(6, n_side=16, box=50.3, rCut=12.0, rSwitch=10.0, beta=0.32)
    tiles = {}
    for s in (small, large):
        nb = NbDirect(s)
        pos = nb.positions_tensor()
        nb.update_domdec(pos, True)
        tiles[s.N] = nb.tuning()["tiles_per_work"]
        a = nb.evaluate(pos)[0]
        nb.set_tuning(8)                                  # the general setting: the list stays valid
        assert torch.equal(a, nb.evaluate(pos)[0])
        nb.close()
    assert tiles[small.N] == 2 and tiles[large.N] == 8
    # together: each replica's bits are those it has alone
    pair = [small, systems.water_box(7)]
    nb = NbDirect(pair)
    pos = nb.positions_tensor()
    nb.update_domdec(pos, True)
    f = nb.evaluate(pos)[0]
    for r, s in enumerate(pair):
        one = NbDirect(s)
        p = one.positions_tensor()
        one.update_domdec(p, True)
        assert torch.equal(f[nb.starts[r]:nb.starts[r + 1]], one.evaluate(p)[0])
        one.close()
    nb.close()


def _msld_of_waters(seed):
    """A water box whose first six molecules are the blocks of two sites (few
    types, so the LJ table is in shared memory alone and in a batch)."""
    s = systems.water_box(seed)
    s.msld = systems._msld_layout(np.random.default_rng(seed), [3, 3])
    s.nbonds = s.nbonds.copy()
    for b in range(1, 7):
        s.nbonds["siteBlock"][3 * (b - 1):3 * b] = (int(s.msld.lambdaSite[b]) << 16) | b
    return s


@pytest.mark.parametrize("methods", [(e, v) for e in range(3) for v in range(3)])
@pytest.mark.parametrize("n_side", [6, 16])
def test_water_beside_msld_replica_keeps_its_bits(cuda, n_side, methods):
    """The kernel of a batch with MSLD replicas sums a replica without MSLD
    atoms in the order of the kernel that it runs in alone."""
    water = systems.water_box(5, n_side=n_side, box=n_side * 18.856 / 6)
    pair = [water, _msld_of_waters(9)]
    for s in pair:
        s.elecMethod, s.vdwMethod = methods
    nb = NbDirect(pair)
    pos, lam = nb.positions_tensor(), nb.lambdas_tensor()
    nb.update_domdec(pos, True)
    f, l, e = nb.evaluate(pos, lam)
    f1 = nb.evaluate(pos, lam, calc_energy=False)[0]
    for r, s in enumerate(pair):
        one = NbDirect(s)
        p = one.positions_tensor()
        one.update_domdec(p, True)
        g, m, d = one.evaluate(p)
        at = slice(nb.starts[r], nb.starts[r + 1])
        assert torch.equal(f[at], g) and float(e[r]) == float(d[0])
        assert torch.equal(f1[at], one.evaluate(p, calc_energy=False)[0])
        assert torch.equal(l[nb.lam_starts[r]:nb.lam_starts[r + 1]], m)
        one.close()
    nb.close()


def test_tuning_reports_the_list_in_use(cuda):
    """Naming the general default after a default build keeps that list, and its
    split is the one reported; the next build has the bits of a handle tuned
    before its first."""
    s = systems.water_box(5)
    nb = NbDirect(s)
    pos = nb.positions_tensor()
    nb.update_domdec(pos, True)
    work = nb.list_sizes()["work"]
    nb.set_tuning(8, 2)
    assert nb.tuning() == {"tiles_per_work": 2, "ctas_per_sm": 2, "tail_items": 0}
    nb.evaluate(pos)
    assert nb.list_sizes()["work"] == work
    nb.set_tuning(8, 2)                                   # once more: nothing changes
    nb.evaluate(pos)
    nb.update_domdec(pos, True)
    assert nb.tuning() == {"tiles_per_work": 8, "ctas_per_sm": 2, "tail_items": 2}
    one = NbDirect(s)
    one.set_tuning(8)
    assert one.tuning() == {"tiles_per_work": 8, "ctas_per_sm": 0, "tail_items": 2}
    one.update_domdec(pos, True)
    assert torch.equal(nb.evaluate(pos)[0], one.evaluate(pos)[0])
    nb.set_tuning(4, 2)                                   # any other change asks for a rebuild
    assert nb.tuning()["tiles_per_work"] == 4
    with pytest.raises(Exception):
        nb.evaluate(pos)
    nb.close()
    one.close()


@pytest.mark.parametrize("r", [0.12, 0.2, 0.4])
@pytest.mark.parametrize("pick", [(1, 302), (2, 500)])
def test_pair_energies_beyond_the_fast_range(cuda, pick, r):
    """Hydrogens of two molecules close enough for pair energies of some hundreds
    to 4e5: with the ordinary ones they share a step, whose sum switches to the
    general conversion at 1000."""
    s = systems.water_box(8)
    x = s.xyz.copy()
    i, j = pick
    mol = 3 * (j // 3)
    x[mol:mol + 3] += x[i] + np.float32([r, 0, 0]) - x[j]  # the whole molecule of j beside i
    s.xyz = x
    nb = NbDirect(s)
    pos = nb.positions_tensor()
    nb.update_domdec(pos, True)
    _, _, e = nb.evaluate(pos)
    o = oracle.nbdirect(s)
    assert nb.status() == 0
    # FP32 coordinates decide the distance: the oracle sees the same ones
    assert abs(float(e[0]) - o["energy"]) <= TOL * max(abs(o["energy"]), s.N)
    nb.close()
