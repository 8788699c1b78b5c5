"""Handles of different sizes driven by several host threads at once: a handle's
launches do not depend on what another thread's handle needs."""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

from blade_b200 import _lib, systems
from blade_b200.nbdirect import NbDirect

pytestmark = pytest.mark.gpu


def _msld(seed, subs):
    """Alchemical box with `subs` substituents at each of three sites: the pair
    kernel's shared memory grows with their number."""
    return systems.msld_water(seed, 3, subs)


def test_handles_of_different_sizes_in_two_threads(cuda):
    handles = []
    for reps in ([_msld(9, 4)], [_msld(9, 4), _msld(10, 4)]):
        nb = NbDirect(reps)
        pos, lam = nb.positions_tensor(), nb.lambdas_tensor()
        nb.update_domdec(pos, True)
        handles.append((nb, pos, lam, nb.evaluate(pos, lam, calc_energy=False)[0]))
    torch.cuda.synchronize()
    lib = _lib.lib()
    start = threading.Barrier(len(handles))
    results = [None] * len(handles)

    def work(k):
        nb, pos, lam, ref = handles[k]
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            f = torch.zeros_like(ref)
        stream.synchronize()
        out = _lib.Outputs(force64=f.data_ptr())
        boxes = np.ascontiguousarray(nb.boxes)
        args = (nb.h, C.c_void_p(pos.data_ptr()), C.c_void_p(lam.data_ptr()), boxes.ctypes.data_as(C.c_void_p),
                _lib.BNB_OUT_SET, C.byref(out), C.c_void_p(stream.cuda_stream))
        start.wait()
        codes = [lib.bnb_compute(*args) for _ in range(3000)]
        stream.synchronize()
        results[k] = (set(codes), torch.equal(f, ref))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(handles))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert results == [({0}, True)] * len(handles)
    for h in handles:
        h[0].close()
