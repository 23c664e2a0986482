"""The fused even/odd launch of the AA rows (csrc/lbm_pair.cuh) where it
has to wait: lattices with more tiles than the lead of the even steps, so that
blocks run the even step of one tile and the odd step of another while the
steps they depend on are still under way. Small lattices, whose odd steps all
follow the even ones, are in test_gpu_parity.py. The reference is the same
lattice as two x-slabs, which take one launch per step; the arithmetic is the
same, so the fields agree bit for bit in every storage."""
import numpy as np
import pytest

import lbmb200
from lbm_cases import random_pdfs
from test_gpu_slabs import _run_slabs

pytestmark = pytest.mark.gpu


def _spheres(dims, porosity):
    return lbmb200.spheres(dims, 42, porosity, 3.0, 6.0, 4000)[0]


CASES = [
    # periodic rings: the first x plane's odd step needs the last plane's even step
    (lambda: _spheres((160, 61, 60), 0.6), ["-precision", "fp64"]),
    (lambda: _spheres((160, 61, 60), 0.6), ["-precision", "fp32"]),
    (lambda: _spheres((160, 61, 60), 0.6), ["-precision", "fp16"]),
    (lambda: lbmb200.geometry("fluid", (131, 41, 43), (1, 1, 1)), ["-pad", "no"]),
    # numberings whose neighbours lie further apart, and closed x ends
    (lambda: _spheres((150, 48, 50), 0.6), ["-blk", "24"]),
    (lambda: lbmb200.geometry("box", (120, 44, 45), (0, 1, 1)), ["-blk-z", "16"]),
    # planes of less than one tile
    (lambda: lbmb200.geometry("fluid", (2500, 9, 11), (1, 1, 1)), ["-pad", "no"]),
]


@pytest.mark.parametrize("make,kargs", CASES)
def test_fused_pairs_equal_separate_steps(make, kargs):
    lat = make()
    init = random_pdfs(lat.mask.size, 53)
    cd = lbmb200.case(omega=1.2, xforce=2e-4, iterations=8)
    kargs = ["-lambda", "3/16"] + kargs
    inst = lbmb200.kernel("cuda-list-aa-pv-soa").init(lat, kernel_args=kargs)
    try:
        assert inst.launches_for(2) == 1 and lat.n_fluid > 450 * 256
        inst.set_field(init)
        inst.run(cd)
        whole = inst.get_field()
    finally:
        inst.deinit()
    got = _run_slabs(lat, 2, init, cd, 4, layout="list", kargs=kargs)
    m = lat.mask != 0
    assert np.array_equal(got[m], whole[m])


AA_CASES = [
    (lambda: lbmb200.geometry("fluid", (40, 61, 59), (1, 1, 1))),
    (lambda: lbmb200.geometry("channel", (45, 70, 64), (1, 0, 0))),
    (lambda: lbmb200.geometry("channel", (70, 50, 49), (0, 0, 0))),   # open x faces
    (lambda: lbmb200.geometry("fluid", (30, 66, 67), (0, 1, 0))),     # open and periodic faces
    (lambda: _spheres((60, 47, 53), 0.5)),
    # planes in strips, with and without tiles that need the next strip through a periodic face
    (lambda: lbmb200.geometry("fluid", (9, 330, 310), (1, 1, 1))),
    (lambda: lbmb200.geometry("channel", (10, 317, 331), (1, 0, 0))),
    # rows longer than a tile, planes of one tile
    (lambda: lbmb200.geometry("fluid", (5, 150, 700), (1, 0, 1))),
    (lambda: lbmb200.geometry("fluid", (900, 11, 13), (1, 1, 1))),
]


@pytest.mark.parametrize("make", AA_CASES)
def test_fused_full_array_pairs_equal_separate_steps(make):
    lat = make()
    init = random_pdfs(lat.mask.size, 59)
    cd = lbmb200.case(omega=1.2, xforce=2e-4, iterations=8)
    inst = lbmb200.kernel("cuda-aa-soa").init(lat, kernel_args=["-lambda", "3/16"])
    try:
        assert inst.launches_for(2) == 1 and inst.launches_for(7) == 4
        inst.set_field(init)
        inst.run(cd)
        whole = inst.get_field()
    finally:
        inst.deinit()
    got = _run_slabs(lat, 2, init, cd, 4)
    m = lat.mask != 0
    assert np.array_equal(got[m], whole[m])


def test_slab_steps_on_a_whole_lattice():
    """The slab entry points step a whole-lattice instance half by half; fused
    pairs before and after them continue the same run."""
    import ctypes
    lat = lbmb200.geometry("blocks-4", (30, 26, 25), (1, 1, 1))
    init = random_pdfs(lat.mask.size, 61)
    cd = lbmb200.case(omega=1.1, xforce=2e-4, iterations=4)
    fields = []
    L = lbmb200.lib()
    for halves in (False, True):
        inst = lbmb200.kernel("cuda-aa-soa").init(lat, kernel_args=["-lambda", "3/16"])
        try:
            inst.set_field(init)
            inst.run(cd)
            if halves:
                for half in (0, 1, 0, 1):
                    assert L.lbm_aa_slab_step(inst.kdp, ctypes.byref(cd), half, None) == 0
                inst.sync_mirror()
            else:
                inst.run(cd)
            inst.run(cd)
            fields.append(inst.get_field())
        finally:
            inst.deinit()
    m = lat.mask != 0
    assert np.array_equal(fields[0][m], fields[1][m])


@pytest.mark.parametrize("kname,prec", [("cuda-list-aa-pv-soa", "fp64"), ("cuda-list-aa-pv-soa", "fp32"),
                                        ("cuda-list-pull-soa", "fp64"), ("cuda-aa-soa", "fp64")])
@pytest.mark.parametrize("dims", [(65, 64, 63), (128, 128, 64), (129, 127, 64), (256, 128, 128), (257, 128, 129)])
def test_every_group_size(kname, prec, dims):
    """Either side of the tile counts at which the groups grow, whole and
    ragged last groups: the fused steps against separate ones."""
    lat = lbmb200.geometry("fluid", dims, (1, 1, 1))
    init = random_pdfs(lat.mask.size, 29)
    cd = lbmb200.case(omega=1.2, xforce=2e-4, iterations=4)
    kargs = ["-lambda", "3/16"] + (["-precision", prec] if "list" in kname else [])
    inst = lbmb200.kernel(kname).init(lat, kernel_args=kargs)
    try:
        assert inst.launches_for(4) == 2
        inst.set_field(init)
        inst.run(cd)
        whole = inst.get_field()
        if "pull" in kname:
            inst.set_field(init)
            for _ in range(4):
                inst.run(lbmb200.case(omega=1.2, xforce=2e-4, iterations=1))
            apart = inst.get_field()
    finally:
        inst.deinit()
    if "pull" not in kname:
        apart = _run_slabs(lat, 2, init, cd, 2, layout="list" if "list" in kname else "full", kargs=kargs)
    assert np.array_equal(apart, whole)


@pytest.mark.parametrize("prec", ["fp64", "fp32", "fp16"])
@pytest.mark.parametrize("dims,steps", [((9, 8, 7), 2), ((30, 27, 29), 9), ((47, 44, 45), 6)])
def test_small_domains_in_one_launch(prec, dims, steps):
    """Domains whose tiles are all resident take many pairs per launch; one
    tile, a part tile, several blocks, odd step counts (rounded up to pairs)."""
    lat = _spheres(dims, 0.6) if dims[0] > 9 else lbmb200.geometry("fluid", dims, (1, 1, 1))
    init = random_pdfs(lat.mask.size, 67)
    cd = lbmb200.case(omega=1.2, xforce=2e-4, iterations=steps)
    kargs = ["-lambda", "3/16", "-precision", prec]
    inst = lbmb200.kernel("cuda-list-aa-pv-soa").init(lat, kernel_args=kargs)
    try:
        assert inst.launches_for(steps) == 1
        inst.set_field(init)
        inst.run(cd)
        assert inst.last_launches == 1
        inst.run(cd)
        whole = inst.get_field()
    finally:
        inst.deinit()
    got = _run_slabs(lat, 2, init, cd, 2 * ((steps + 1) // 2), layout="list", kargs=kargs)
    m = lat.mask != 0
    assert np.array_equal(got[m], whole[m])


def test_captured_steps_replay():
    """A captured sequence of fused pairs can be replayed: the launches count
    themselves on the device."""
    import ctypes

    import torch
    cd = lbmb200.case(omega=1.1, xforce=1e-4, iterations=4)
    L = lbmb200.lib()
    for lat in (_spheres((130, 44, 40), 0.6), _spheres((30, 27, 29), 0.6)):
        init = random_pdfs(lat.mask.size, 71)
        fields = []
        for replay in (False, True):
            inst = lbmb200.kernel("cuda-list-aa-pv-soa").init(lat, kernel_args=["-lambda", "3/16"])
            try:
                inst.set_field(init)
                inst.run(cd)
                if replay:
                    st = ctypes.c_void_p()
                    assert L.lbm_b200_device_state(inst.kdp, None, None, None, ctypes.byref(st)) == 0
                    stream = torch.cuda.ExternalStream(st.value)
                    g = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(g, stream=stream):
                        inst.step_device(cd, 4)
                    for _ in range(3):
                        g.replay()
                    torch.cuda.synchronize()
                    inst.sync_mirror()
                else:
                    inst.run(lbmb200.case(omega=1.1, xforce=1e-4, iterations=12))
                fields.append(inst.get_field())
            finally:
                inst.deinit()
        m = lat.mask != 0
        assert np.array_equal(fields[0][m], fields[1][m])


TWO_GRID_CASES = [
    ("cuda-list-pull-soa", lambda: _spheres((140, 62, 60), 0.6)),
    ("cuda-list-pull-split-nt-2s-soa", lambda: lbmb200.geometry("fluid", (131, 47, 46), (1, 0, 1))),
    ("cuda-list-push-soa", lambda: _spheres((140, 62, 60), 0.6)),
] + [(k, g) for k in ("cuda-push-soa", "cuda-pull-soa") for g in (
    lambda: lbmb200.geometry("fluid", (60, 61, 59), (1, 1, 1)),
    lambda: lbmb200.geometry("channel", (45, 70, 64), (1, 0, 0)),
    lambda: lbmb200.geometry("channel", (70, 50, 49), (0, 0, 0)),
    lambda: lbmb200.geometry("fluid", (30, 66, 67), (0, 1, 0)),
    lambda: lbmb200.geometry("fluid", (7, 5, 300), (1, 0, 0)),
    lambda: _spheres((60, 47, 53), 0.5),
    lambda: lbmb200.geometry("channel", (10, 317, 331), (1, 0, 0)))]


@pytest.mark.parametrize("kname,make", TWO_GRID_CASES)
def test_two_grid_steps_in_one_launch(kname, make):
    """Two steps per launch (and a single last one) against one launch per
    step: one-step runs take the latter."""
    lat = make()
    init = random_pdfs(lat.mask.size, 73)
    fields = []
    for steps in ([7], [1] * 7):
        inst = lbmb200.kernel(kname).init(lat, kernel_args=["-lambda", "3/16"])
        try:
            assert inst.launches_for(7) == 4 and inst.launches_for(1) == 1
            inst.set_field(init)
            for n in steps:
                inst.run(lbmb200.case(omega=1.2, xforce=2e-4, iterations=n))
            fields.append(inst.get_field())
        finally:
            inst.deinit()
    m = lat.mask != 0
    assert np.array_equal(fields[0][m], fields[1][m])


@pytest.mark.parametrize("parts", [False, True])
def test_first_half_steps_on_a_callers_stream(parts):
    """The first half steps of a whole-lattice instance may go to any stream."""
    import ctypes

    import torch
    lat = lbmb200.geometry("blocks-4", (30, 26, 25), (1, 1, 1))
    init = random_pdfs(lat.mask.size, 79)
    cd = lbmb200.case(omega=1.1, xforce=2e-4, iterations=4)
    L = lbmb200.lib()
    fields = []
    for apart in (False, True):
        inst = lbmb200.kernel("cuda-aa-soa").init(lat, kernel_args=["-lambda", "3/16"])
        try:
            inst.set_field(init)
            if apart:
                mine = torch.cuda.Stream()
                st = ctypes.c_void_p(mine.cuda_stream)
                for half in (0, 1, 0, 1):
                    if parts:
                        step = L.lbm_aa_slab_odd_part if half else L.lbm_aa_slab_even_part
                        assert all(step(inst.kdp, ctypes.byref(cd), k, st) == 0 for k in (0, 1))
                    else:
                        assert L.lbm_aa_slab_step(inst.kdp, ctypes.byref(cd), half, st) == 0
                mine.synchronize()
                inst.sync_mirror()
            else:
                inst.run(cd)
            fields.append(inst.get_field())
        finally:
            inst.deinit()
    m = lat.mask != 0
    assert np.array_equal(fields[0][m], fields[1][m])
