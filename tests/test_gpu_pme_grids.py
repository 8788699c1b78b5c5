"""Own PME transforms over lengths of every radix, odd and even, unequal edges,
and the hand-over to cuFFT outside their range, against the FP64 oracle."""
import dataclasses

import numpy as np
import pytest
import torch

from blade_b200 import systems
from blade_b200.nbdirect import NbDirect
from oracle import pme_oracle

pytestmark = pytest.mark.gpu

# radices 2-8 alone and mixed, odd rows without a partner, odd z (no Nyquist),
# one-CTA planes up to the shared-memory limit; 7 and 200 go to cuFFT
GRIDS = [(6, 6, 6), (8, 9, 10), (15, 16, 18), (18, 15, 25), (20, 20, 20), (27, 27, 27), (32, 24, 40), (36, 45, 48),
         (54, 54, 54), (64, 64, 64), (30, 81, 75), (128, 20, 16), (16, 128, 128), (20, 144, 144), (16, 162, 160),
         (300, 8, 8), (14, 20, 20), (20, 20, 28), (8, 200, 200)]


def _run(nb, energy=True):
    pos, lam = nb.positions_tensor(), nb.lambdas_tensor()
    nb.update_domdec(pos, True)
    f, l, e = nb.evaluate_pme(pos, lam, energy)
    g, _, _ = nb.evaluate_pme(pos, lam, energy)              # the charge grid was left cleared
    assert torch.equal(f, g)
    return f.cpu().numpy(), l.cpu().numpy(), e.cpu().numpy()


@pytest.mark.parametrize("grid", GRIDS)
def test_grids_against_oracle(cuda, grid):
    s = systems.msld_water(21)
    nb = NbDirect(s)
    nb.set_pme(6, grid=[grid])
    f, l, e = _run(nb)
    lam = nb.lambdas_tensor().cpu().numpy().astype(np.float64)
    eo, go, lo, _ = pme_oracle.pme_recip(s.xyz, s.nbonds["q"], s.box, grid, 6, float(np.float32(s.betaEwald)),
                                         float(np.float32(systems.KELEC_AKMA)), s.nbonds["siteBlock"], lam)
    nb.close()
    # FP32 grid and transforms: errors of a few 2^-24 of the largest potential term
    assert np.sqrt(((f - go) ** 2).sum()) <= 1e-5 * np.sqrt((go ** 2).sum())
    assert abs(e[0] - eo) <= 1e-5 * abs(eo)
    assert np.abs(l[1:] - lo[1:]).max() <= 1e-5 * np.abs(lo).max()


def test_mixed_sizes_in_one_handle(cuda):
    """Replicas of different sizes share the three launches and give the bits of each alone."""
    reps = [systems.msld_water(30 + k) for k in range(3)]
    big = dataclasses.replace(reps[1], box=np.float32([24.0, 20.0, 30.0]))
    reps[1] = big
    nb = NbDirect(reps)
    nb.set_pme(6)
    assert nb.pme_grid(0) != nb.pme_grid(1)
    f, l, e = _run(nb)
    for r, s in enumerate(reps):
        one = NbDirect(s)
        one.set_pme(6)
        f1, l1, e1 = _run(one)
        assert np.array_equal(f[nb.starts[r]:nb.starts[r + 1]], f1) and e[r] == e1[0]
        one.close()
    nb.close()


@pytest.mark.parametrize("order", [4, 6, 8])
@pytest.mark.parametrize("side,box", [(1, 12.0), (2, 12.0), (15, 47.14), (16, 50.28)])
def test_sizes_of_the_spread_and_gather(cuda, order, side, box):
    """A few atoms, and both sides of the line between small and large warps' shares (10,656 and 9,472 atoms)."""
    s = systems.water_box(9, n_side=side, box=box, rCut=6.0, rSwitch=5.0)
    if side == 16:
        s = dataclasses.replace(s, xyz=s.xyz[:-2], nbonds=s.nbonds[:-2], excl=s.excl[(s.excl < s.N - 2).all(1)])
    nb = NbDirect(s)
    nb.set_pme(order, grid=[(32, 32, 32)])
    f, _, e = _run(nb)
    eo, go, _, _ = pme_oracle.pme_recip(s.xyz, s.nbonds["q"], s.box, (32, 32, 32), order,
                                        float(np.float32(s.betaEwald)), float(np.float32(systems.KELEC_AKMA)))
    nb.close()
    # FP32 grid values: relative to the scale of the largest terms, which cancel in few waters
    assert np.sqrt(((f - go) ** 2).sum()) <= 2e-5 * max(np.sqrt((go ** 2).sum()), 1e-2)
    assert abs(e[0] - eo) <= 2e-5 * max(abs(eo), s.N)


@pytest.mark.parametrize("grids", [[(96, 96, 96), (80, 100, 96)], [(162, 30, 32), (32, 30, 18)], [(162, 100, 100)],
                                   [(48, 48, 48)] * 3 + [(640, 16, 16)]])
def test_launch_shapes_keep_the_bits(cuda, grids):
    """More planes than SMs and long edges change the threads of a CTA (fewer a
    plane, more a tile of columns), not the results."""
    reps = [systems.msld_water(30 + k % 2) for k in range(len(grids))]
    nb = NbDirect(reps)
    nb.set_pme(6, grid=grids)
    f, l, e = _run(nb)
    lam = nb.lambdas_tensor().cpu().numpy().astype(np.float64)
    for r, s in enumerate(reps):
        one = NbDirect(s)
        one.set_pme(6, grid=[grids[r]])
        f1, l1, e1 = _run(one)
        one.close()
        at = slice(nb.starts[r], nb.starts[r + 1])
        assert np.array_equal(f[at], f1) and e[r] == e1[0]
        eo, go, _, _ = pme_oracle.pme_recip(s.xyz, s.nbonds["q"], s.box, grids[r], 6, float(np.float32(s.betaEwald)),
                                            float(np.float32(systems.KELEC_AKMA)), s.nbonds["siteBlock"],
                                            lam[nb.lam_starts[r]:nb.lam_starts[r + 1]])
        assert np.sqrt(((f[at] - go) ** 2).sum()) <= 1e-5 * np.sqrt((go ** 2).sum())
        assert abs(e[r] - eo) <= 1e-5 * abs(eo)
    nb.close()
