"""CPU tests of the product's host layer: the C ABI library loads and exports
every function include/lbm_b200.h declares; geometry masks and list layouts
(numbering, padding, adjacency) equal the oracle's and the reference's bit for
bit. No GPU is touched: these calls never reach the CUDA runtime."""
import os
import re

import numpy as np
import pytest

import lbmb200
from lbm_cases import FIELD_CASES

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_functions():
    names = []
    for fn in sorted(os.listdir(os.path.join(ROOT, "include"))):
        if not fn.endswith(".h"):
            continue
        text = open(os.path.join(ROOT, "include", fn)).read()
        text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
        for m in re.finditer(r"^[A-Za-z_][\w\s\*]*?\b([A-Za-z_]\w*)\s*\([^;{]*\)\s*;", text, flags=re.M):
            if m.group(0).lstrip().startswith(("typedef", "void (*", "return")):
                continue
            names.append(m.group(1))
    return sorted(set(names))


def test_library_exports_every_declared_function():
    names = _declared_functions()
    assert "D3Q19CudaAaInit_AaSoA" in names and "lbm_b200_kernels" in names
    lib = lbmb200.lib()
    missing = [n for n in names if not hasattr(lib, n)]
    assert not missing, missing


def test_kernel_table_names():
    assert lbmb200.kernel_names() == ["cuda-aa-soa", "cuda-list-aa-pv-soa",
                                      "cuda-list-pull-split-nt-1s-soa", "cuda-list-pull-split-nt-2s-soa",
                                      "cuda-list-aa-soa", "cuda-list-aa-ria-soa", "cuda-list-push-soa",
                                      "cuda-list-pull-soa", "cuda-push-soa", "cuda-pull-soa"]
    # case-insensitive lookup as src/Main.c:543
    assert lbmb200.kernel("CUDA-AA-SOA").name == "cuda-aa-soa"
    with pytest.raises(KeyError):
        lbmb200.kernel("aa-soa")


GEOMS = ["box", "channel", "pipe", "blocks", "blocks-3", "fluid"]
PERIODIC = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 1), (1, 1, 1), (0, 0, 1)]
DIMS = [(16, 16, 16), (17, 9, 13), (7, 9, 8), (1, 4, 5)]


@pytest.mark.parametrize("geo", GEOMS)
@pytest.mark.parametrize("per", PERIODIC)
@pytest.mark.parametrize("dims", DIMS)
def test_geometry_matches_oracle(oracle, geo, per, dims):
    bs = 8 if geo == "blocks" else (3 if geo == "blocks-3" else 0)
    if bs and bs > min(dims) // 2:
        with pytest.raises(ValueError):
            lbmb200.geometry(geo, dims, per)
        return
    lat = lbmb200.geometry(geo, dims, per)
    mask, info = oracle.geometry(geo, dims, per)
    assert np.array_equal(lat.mask, mask)
    assert lat.n_fluid == info["nFluid"]
    assert lat.periodic == info["ldPeriodic"]
    bits = info["geoPeriodicBits"]
    assert lat.geo_periodic == (bits & 1, (bits >> 1) & 1, (bits >> 2) & 1)


def test_geometry_rejects_unknown():
    with pytest.raises(ValueError):
        lbmb200.geometry("sphere", (8, 8, 8))


LAYOUTS = [(g, d, p) for g, d, p in FIELD_CASES] + [("fluid", (3, 3, 3), (1, 1, 1)), ("box", (1, 4, 5), (1, 1, 1))]


@pytest.mark.parametrize("pull", [0, 1])
@pytest.mark.parametrize("blk,pad", [((0, 0, 0), None), ((7, 7, 7), None), ((3, 0, 5), "no"),
                                     ((0, 0, 0), "4096+64,256+8")])
@pytest.mark.parametrize("geo,dims,per", LAYOUTS)
def test_list_layout_matches_oracle(oracle, pull, blk, pad, geo, dims, per):
    lat = lbmb200.geometry(geo, dims, per)
    g1, a1, nf1, nc1 = lbmb200.list_build(lat, pull, blk, pad)
    pad_mode = 0 if pad is None else (1 if pad == "no" else 2)
    if pad_mode == 2:
        expect_nc = oracle.lib.orc_pad_cells  # explicit pairs: compare the count through the C oracle
        import ctypes
        mods = (ctypes.c_int * 2)(4096, 256)
        offs = (ctypes.c_int * 2)(64, 8)
        nc_o = expect_nc(lat.n_fluid, 8, 2, 2, mods, offs)
        if pull:
            nc_o = nc_o + (8 - nc_o % 8)
        assert nc1 == nc_o
        # adjacency with that nCells: rebuild the oracle layout with no padding and re-encode
        g2, a2, nf2, nc2 = oracle.list_layout(pull, dims, lat.periodic, lat.mask, blk, 1)
        d2, n2 = a2 // nc2, a2 % nc2
        a2 = (d2 * nc1 + n2).astype(np.uint32)
    else:
        g2, a2, nf2, nc2 = oracle.list_layout(pull, dims, lat.periodic, lat.mask, blk, pad_mode)
        assert nc1 == nc2
    assert nf1 == nf2 == lat.n_fluid
    assert np.array_equal(g1, g2)
    assert np.array_equal(a1, a2)


@pytest.mark.parametrize("pull", [0, 1])
@pytest.mark.parametrize("geo,dims,per", FIELD_CASES[:5])
def test_list_layout_matches_reference(reference, pull, geo, dims, per):
    lat = lbmb200.geometry(geo, dims, per)
    kernel = "list-pull-split-nt-1s-soa" if pull else "list-aa-pv-soa"
    g1, a1, nf1, nc1 = lbmb200.list_build(lat, pull)
    g2, a2, nf2, nc2 = reference.list_layout(kernel, dims, lat.periodic, lat.mask)
    assert (nf1, nc1) == (nf2, nc2)
    assert np.array_equal(g1, g2)
    assert np.array_equal(a1, a2)


def test_pad_strings():
    L = lbmb200.lib()
    assert L.lbmh_pad_cells(3584, 8, None) == 3584 + 260624
    assert L.lbmh_pad_cells(3584, 8, b"auto") == 3584 + 260624
    assert L.lbmh_pad_cells(1000, 8, b"no") == 1000
    assert L.lbmh_pad_cells(1000, 8, b"64+8") == 1001  # to the next multiple of 8 cells, plus one
    assert L.lbmh_pad_cells(1000, 8, b"64+64") == -1   # offset >= modulus is rejected
    assert L.lbmh_pad_cells(1000, 8, b"abc") == -1


@pytest.mark.parametrize("pull", [0, 1])
def test_packing_layout_matches_reference(reference, pull):
    # a seeded periodic sphere packing (r in [6, 12], porosity 0.40): the host
    # builder's numbering and adjacency equal the reference's Init bit for bit
    lat, _ = lbmb200.spheres((64, 64, 64), 20251203, 0.40, 6.0, 12.0)
    kernel = "list-pull-split-nt-1s-soa" if pull else "list-aa-pv-soa"
    g1, a1, nf1, nc1 = lbmb200.list_build(lat, pull)
    g2, a2, nf2, nc2 = reference.list_layout(kernel, lat.dims, lat.periodic, lat.mask)
    assert (nf1, nc1) == (nf2, nc2) == (lat.n_fluid, nc2)
    assert np.array_equal(g1, g2)
    assert np.array_equal(a1, a2)


@pytest.mark.slow
@pytest.mark.parametrize("pull", [0, 1])
def test_packing_256_layout_matches_reference_fixture(pull):
    # the 256^3 packing of the throughput workload: the host builder's layout
    # hashes equal those of the reference's Init (tests/golden/packing256.json,
    # written by tests/golden/make_packing_golden.py)
    import hashlib
    import json
    path = os.path.join(ROOT, "tests", "golden", "packing256.json")
    with open(path) as f:
        meta = json.load(f)
    lat, _ = lbmb200.spheres((meta["edge"],) * 3, meta["seed"], 0.40, 6.0, 12.0)
    assert hashlib.sha256(lat.mask.tobytes()).hexdigest() == meta["mask_sha256"]
    lay = meta["layouts"]["pull" if pull else "push"]
    g, a, nf, nc = lbmb200.list_build(lat, pull)
    assert (nf, nc) == (lay["n_fluid"], lay["n_cells"])
    assert hashlib.sha256(g.tobytes()).hexdigest() == lay["grid_sha256"]
    assert hashlib.sha256(a.tobytes()).hexdigest() == lay["adj_sha256"]


def _field_inputs():
    import pandas
    import torch
    row = np.arange(19.0) / 7
    full = np.arange(12 * 19.0).reshape(12, 19)
    rows = np.broadcast_to(row, (12, 19))
    return {
        "array": full, "flat": full.reshape(-1), "float32": full.astype(np.float32), "transposed": full.T.copy().T,
        "nested list": full.tolist(), "tensor": torch.from_numpy(full), "tensor float32": torch.from_numpy(full).float(),
        "tensor repeated row": torch.from_numpy(row).expand(12, 19), "data frame": pandas.DataFrame(full),
        "memory view": memoryview(full), "memory view of a repeated row": memoryview(rows), "repeated row": rows,
        "repeated float32 row": np.broadcast_to(row.astype(np.float32), (12, 19)),
        "repeated number": np.broadcast_to(np.float64(0.5), (12, 19)),
    }


@pytest.mark.parametrize("name", [
    "array", "flat", "float32", "transposed", "nested list", "tensor", "tensor float32", "tensor repeated row",
    "data frame", "memory view", "memory view of a repeated row", "repeated row", "repeated float32 row",
    "repeated number"])
def test_set_field_takes_what_numpy_takes(name, monkeypatch):
    """Instance.set_field hands the library the cells' PDFs, whatever kind of
    array they come in; a repeated row may go by itself."""
    import ctypes
    import types
    pdfs = _field_inputs()[name]
    got = []

    def taken(n):
        return lambda kdp, ld, p: got.append(np.broadcast_to(np.ctypeslib.as_array(p, shape=(n, 19)), (12, 19)).copy())

    fake = types.SimpleNamespace(lbm_b200_set_field=taken(12), lbm_b200_set_uniform=taken(1))
    monkeypatch.setattr(lbmb200, "lib", lambda: fake)
    lattice = types.SimpleNamespace(mask=np.ones(12, np.int32), desc=ctypes.c_int(0))
    lbmb200.Instance(None, lattice, None).set_field(pdfs)
    assert len(got) == 1 and np.array_equal(got[0], np.ascontiguousarray(pdfs, dtype=np.float64).reshape(12, 19))
