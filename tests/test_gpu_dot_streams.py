"""dot and nrm2 share their scratch per device: calls that follow one another on
different streams, and calls of several host threads, each return their own sum."""
import ctypes as C
import threading

import numpy as np
import pytest

from senk_gb300 import lib as L

pytestmark = pytest.mark.gpu

SIZES = [1, 255, 257, 4096, 16384, 300_001]


def _data(seed):
    import torch
    rng = np.random.default_rng(seed)
    x = [rng.integers(-8, 9, n).astype(np.float64) for n in SIZES]      # sums of integers: exact in any order
    y = [rng.integers(-8, 9, n).astype(np.float64) for n in SIZES]
    dev = [(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()) for a, b in zip(x, y)]
    return dev, [float(a @ b) for a, b in zip(x, y)], [float(np.sqrt(a @ a)) for a in x]


def _loop(dev, dots, nrms, streams, rounds, bad):
    r = C.c_double()
    for i in range(rounds):
        k = (7 * i + i // 5) % len(SIZES)
        s = streams[i % len(streams)].cuda_stream
        x, y = dev[k]
        if L.lib().senk_dev_dot_d(x.data_ptr(), y.data_ptr(), SIZES[k], C.byref(r), s) or r.value != dots[k]:
            bad.append(("dot", i, SIZES[k], r.value, dots[k]))
        if i % 3 == 0:
            rc = L.lib().senk_dev_nrm2_d(x.data_ptr(), SIZES[k], C.byref(r), s)
            if rc or r.value != nrms[k]:
                bad.append(("nrm2", i, SIZES[k], r.value, nrms[k]))


def test_alternating_streams():
    import torch
    dev, dots, nrms = _data(1)
    torch.cuda.synchronize()
    bad = []
    _loop(dev, dots, nrms, [torch.cuda.Stream() for _ in range(3)], 3000, bad)
    assert not bad, bad[:3]


def test_host_threads():
    import torch
    data = [_data(s) for s in range(4)]
    torch.cuda.synchronize()
    bad = []
    ts = [threading.Thread(target=_loop, args=(*d, [torch.cuda.Stream(), torch.cuda.Stream()], 1000, bad)) for d in data]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:3]
