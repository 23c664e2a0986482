"""Memory of instances and batches (csrc/lbm_mem.cuh): kept device memory is
reused and given back, new instances start from zeros whatever the memory held
before, and a repeated row sets the same state as the written-out field."""
import threading

import numpy as np
import pytest

import lbmb200
from lbm_cases import W, random_pdfs

pytestmark = pytest.mark.gpu


def _run(kname, lat, init, kargs=()):
    inst = lbmb200.kernel(kname).init(lat, kernel_args=["-lambda", "3/16", *kargs])
    try:
        fresh = inst.get_field()
        if init is not None:
            inst.set_field(init)
        inst.run(lbmb200.case(omega=1.2, xforce=1e-4, iterations=6))
        return fresh, inst.get_field()
    finally:
        inst.deinit()


@pytest.mark.parametrize("kname,kargs", [("cuda-list-aa-pv-soa", ()), ("cuda-list-aa-pv-soa", ("-precision", "fp16")),
                                         ("cuda-aa-soa", ()), ("cuda-pull-soa", ()), ("cuda-list-push-soa", ())])
def test_reused_memory_starts_clean(kname, kargs):
    lat = lbmb200.geometry("fluid", (20, 18, 17), (1, 1, 1))
    init = random_pdfs(lat.mask.size, 5)
    f0, a = _run(kname, lat, init, kargs)
    lbmb200.lib().lbm_b200_release_memory()
    for _ in range(2):
        f1, b = _run(kname, lat, init, kargs)
        assert np.array_equal(a, b) and np.array_equal(f0, f1)


@pytest.mark.parametrize("kname", ["cuda-list-aa-pv-soa", "cuda-list-pull-soa", "cuda-aa-soa", "cuda-pull-soa"])
def test_repeated_row_equals_written_out_field(kname):
    lat = lbmb200.geometry("blocks-3", (13, 11, 12), (1, 0, 1))
    rows = np.broadcast_to(W * 1.01, (lat.mask.size, 19))
    m = lat.mask != 0
    assert np.array_equal(_run(kname, lat, rows)[1][m], _run(kname, lat, np.array(rows))[1][m])


def test_instances_from_several_threads():
    lat = lbmb200.geometry("fluid", (18, 16, 15), (1, 1, 1))
    init = random_pdfs(lat.mask.size, 9)
    want = _run("cuda-list-aa-pv-soa", lat, init)[1]
    got = [None] * 4

    def work(k):
        for _ in range(5):
            got[k] = _run("cuda-list-aa-pv-soa", lat, init)[1]

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(np.array_equal(g, want) for g in got)


@pytest.mark.parametrize("kname", ["cuda-list-aa-pv-soa", "cuda-list-pull-soa"])
@pytest.mark.parametrize("edge", [12, 40])
def test_state_pointers_have_an_ipc_handle(kname, edge):
    """Other processes may open the PDFs that lbm_b200_device_state points to."""
    import ctypes
    rt = pytest.importorskip("cuda.bindings.runtime")
    inst = lbmb200.kernel(kname).init(lbmb200.geometry("fluid", (edge,) * 3, (1, 1, 1)))
    try:
        for _ in range(2):
            p = ctypes.c_void_p()
            assert lbmb200.lib().lbm_b200_device_state(inst.kdp, ctypes.byref(p), None, None, None) == 0
            assert rt.cudaIpcGetMemHandle(p.value)[0] == rt.cudaError_t.cudaSuccess
            inst.step_device(lbmb200.case(omega=1.2, xforce=0.0, iterations=1), 1)
    finally:
        inst.deinit()
