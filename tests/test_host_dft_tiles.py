"""The sigma = 0 mode's direct DFTs of few, long lines: tiles that are not
mostly lines that are not there.  On the stand-in runtime, without a GPU."""
import ctypes as C
import re

import numpy as np
import pytest

import _fake_cuda
from pyflct_gb300.flct import make_params


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    h = _fake_cuda.Host(_fake_cuda.load(tmp_path_factory.mktemp("fake")))
    yield h
    h.close()


@pytest.mark.parametrize("shape", [(1, 10007), (10007, 1), (1, 1000), (3, 30000), (5, 20000), (8, 4096), (9, 10007), (24, 30000), (33, 10007),
                                   (4, 4), (97, 101), (1000, 1200)])
def test_tiles_hold_the_lines_there_are(host, shape):
    nx, ny = shape
    f = [np.zeros(shape) for _ in range(2)]
    o = [np.zeros(1) for _ in range(3)]
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in (*f, *o)]
    rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, 0.0)), p[0], p[1], nx, ny, *p[2:])
    assert rc == 0
    runs = [(re.search(r"k_dft_(?:long|rows)IL\w+?E((?:Li\d+E)*)", x), x.split()) for x in log if "k_dft_" in x]
    assert len(runs) == 4
    # along the fast axis, along the slow one, and back
    for (m, x), (length, lines) in zip(runs, [(ny, nx), (nx, ny), (nx, ny), (ny, nx)]):
        if not m.group(1):  # one output a thread: more than a tile of 8 lines per SM, and one round of blocks
            assert (int(x[2]), int(x[3])) == (-(-length // 256), lines)
            assert lines <= 8 and -(-length // 64) > 152 >= int(x[2]) * lines
            continue
        assert lines > 8 or length <= 64 * 152 or -(-length // 256) * lines > 152
        pairs, per_thread, freqs = (int(v) for v in re.findall(r"Li(\d+)E", m.group(1)))
        wide, deep = 2 * pairs * per_thread, 256 // pairs * freqs
        assert wide <= max(8, 4 * lines) or int(x[2]) <= 152  # or each on an SM of its own
        assert (int(x[2]), int(x[3])) == (-(-length // deep), -(-lines // wide))
