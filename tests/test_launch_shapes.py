"""The FP32 window kernel's two launch shapes (windows per CTA) per box side,
as the autotuner's file chooses between them.  On the stand-in runtime,
without a GPU."""
import ctypes as C
import json

import numpy as np
import pytest

import _fake_cuda
from pyflct_gb300.flct import make_params


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return _fake_cuda.load(tmp_path_factory.mktemp("fake"))


def shape_of(lib, n, form):
    """Threads per CTA of a call's window launch: a frame of 1.5 n a side holds boxes of side n."""
    m = 3 * n // 2
    a = [np.zeros((m, m)) for _ in range(5)]
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in a]
    host = _fake_cuda.Host(lib)
    rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, 31.0, form=form)), p[0], p[1], m, m, *p[2:])
    host.close()
    assert rc == 0
    threads, = [int(x.split()[5]) for x in log if x.startswith("launch") and "k_window_fp32ILi%d" % n in x]
    return threads


def write(path, **entry):
    path.write_text('{"device": "fake", "entries": [\n  %s\n]}\n' % json.dumps(entry))


@pytest.mark.parametrize("n", range(4, 65, 4))
def test_the_two_shapes_differ(lib, n, tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("FLCT_AUTOTUNE_CACHE", str(path))
    got = []
    for v in (0, 1):
        write(path, box=n, form=0, grid_div=1, ns_per_window=1.0, variant=v)
        got.append(shape_of(lib, n, "auto"))
    assert got[0] == shape_of(lib, n, "fp32")
    assert got[0] != got[1] and all(t % n == 0 for t in got)


def test_a_file_of_other_shapes_is_measured_again(lib, tmp_path, monkeypatch):
    """An entry that names the windows per CTA it was measured with holds for these only;
    one that names none (written before they were) is taken as it is."""
    path = tmp_path / "tune.json"
    monkeypatch.setenv("FLCT_AUTOTUNE_CACHE", str(path))
    entry = dict(box=40, form=0, grid_div=1, ns_per_window=1.0, variant=1)
    write(path, **entry)
    old = shape_of(lib, 40, "auto")
    first = shape_of(lib, 40, "fp32")
    assert old != first
    for teams, want in (([first // 40, old // 40], old), ([first // 40, old // 40 + 1], first), ([4, 8], first),
                        ([first // 40], first)):
        write(path, **entry, teams=teams)
        if want == old:
            assert shape_of(lib, 40, "auto") == old
        else:  # no windows in this call: nothing can be measured, the default shape runs
            assert shape_of(lib, 40, "auto") == first, teams


def test_the_file_names_the_shapes(lib, tmp_path, monkeypatch):
    path = tmp_path / "tune.json"
    monkeypatch.setenv("FLCT_AUTOTUNE_CACHE", str(path))
    a = [np.zeros((60, 60)) for _ in range(5)]
    p = [x.ctypes.data_as(C.POINTER(C.c_double)) for x in a]
    host = _fake_cuda.Host(lib)
    lib.fake_int(100)  # windows to measure on
    try:
        rc, log = host.call("velocity", C.byref(make_params(1.0, 1.0, 31.0, form="auto")), p[0], p[1], 60, 60, *p[2:])
    finally:
        lib.fake_int(0)
    host.close()
    assert rc == 0
    seen = {x.split()[1]: int(x.split()[5]) // 40 for x in log if x.startswith("launch") and "k_window_fp32ILi40" in x}
    e, = json.loads(path.read_text())["entries"]
    assert e["box"] == 40 and e["teams"] == [next(t for k, t in seen.items() if "ILi40ELi%dE" % v in k) for v in (0, 1)]
