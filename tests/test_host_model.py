"""The host layer (csrc/lbm_capi.cu, lbm_batch.cu, lbm_mem.cu) on a model of
the CUDA runtime (tests/host_model): order between streams, lifetimes of host
and device memory, and failed allocations, which a GPU that happens to be quick
enough does not show."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lbm-benchmark-kernels_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
MODEL = os.path.join(ROOT, "tests", "host_model")


@pytest.fixture(scope="module")
def cases(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("host_model")
    flags = ["-g", "-O0", "-fsanitize=address", "-fno-omit-frame-pointer", "-fno-pie", "-I" + CUDA + "/include"]
    jobs = [["g++", "-std=c++17", "-x", "c++", *flags, "-c", os.path.join(CSRC, f + ".cu"), "-o", str(d / (f + ".o"))]
            for f in ("lbm_capi", "lbm_batch", "lbm_mem")]
    jobs.append(["gcc", "-std=c99", "-D_POSIX_C_SOURCE=200112L", *flags, "-c", os.path.join(CSRC, "lbm_host.c"), "-o",
                 str(d / "lbm_host.o")])
    jobs.append(["g++", "-std=c++17", *flags, "-c", os.path.join(MODEL, "cases.cpp"), "-o", str(d / "cases.o")])
    running = [subprocess.Popen(j, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True) for j in jobs]
    for p in running:
        out = p.communicate()[0]
        assert p.returncode == 0, out
    # launchers that no case reaches stay undefined
    exe = str(d / "cases")
    subprocess.run(["g++", "-fsanitize=address", "-no-pie", "-Wl,--unresolved-symbols=ignore-all",
                    *[str(d / (f + ".o")) for f in ("lbm_capi", "lbm_batch", "lbm_mem", "lbm_host", "cases")],
                    "-o", exe], check=True)
    return exe


def _run(exe, name):
    p = subprocess.run([exe, name], capture_output=True, text=True, timeout=60,
                       env={**os.environ, "ASAN_OPTIONS": "detect_leaks=0"})
    assert p.returncode == 0, p.stdout + p.stderr[-4000:]


@pytest.mark.parametrize("name", ["first_odd_part", "first_odd_half", "first_even_half", "first_slab_step_captured"])
def test_first_slab_step_on_a_callers_stream(cases, name):
    """The work items of the odd step are there before any half step that a
    caller's stream takes, captured or not."""
    _run(cases, name)


def test_deinit_waits_for_the_instances_own_device(cases):
    """Deinit may be called with another device current (a finaliser thread,
    one process with several devices) while steps are still queued."""
    _run(cases, "deinit_from_another_device")


def test_batch_results_of_a_lost_state_are_refused(cases):
    """Sums, fields and checkpoints read after a step whose wait ran out."""
    _run(cases, "batch_results_of_a_lost_state")


def test_batch_goes_on_when_memory_runs_out(cases):
    """Every allocation of an admission may fail, those of the fused steps'
    tables among them: no step uses tables that were given back."""
    _run(cases, "batch_without_memory")


def test_batch_steps_after_it_was_empty(cases):
    """A step count first asked for while no domain was there."""
    _run(cases, "batch_steps_while_empty")


@pytest.mark.parametrize("kind", ["full", "list", "slab", "list_slab", "batch"])
def test_uploads_outlive_the_call(cases, kind):
    """Init and admission keep the host tables until their copies are done."""
    _run(cases, "uploads_" + kind)


def test_state_pointers_are_blocks_of_their_own(cases):
    """lbm_b200_device_state gives out pointers that cudaIpcGetMemHandle and
    peer access take."""
    _run(cases, "state_pointer_is_a_block")
    _run(cases, "kept_blocks")


def test_batch_tune_keeps_the_fastest(cases):
    """Fused pairs are among what the tuner chooses from."""
    _run(cases, "batch_tune_keeps_the_fastest")


def _extract(path, *starts):
    """The definitions of a source file that begin with the given lines."""
    text = open(path).read()
    out = []
    for start in starts:
        a = text.index(start)
        assert text.find(start, a + 1) < 0, start
        a = max(text.rfind("\n\n", 0, a), text.rfind("\n}\n", 0, a))
        k = text.index("{", text.index(start))
        depth = 0
        for i in range(k, len(text)):
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            if depth == 0:
                break
        out.append(text[a:i + 1].lstrip("}\n") + (";" if text[i + 1] == ";" else ""))
    return "\n".join(out)


def _device_model(tmp_path_factory, name, source):
    """Device code on the host: tests/host_model/NAME.cpp around `source`."""
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp(name)
    (d / "extracted.inc").write_text(source)
    exe = str(d / name)
    p = subprocess.run(["g++", "-std=c++20", "-O1", "-w", "-pthread", "-I" + CUDA + "/include", "-I" + str(d),
                        os.path.join(MODEL, name + ".cpp"), "-o", exe], capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    return exe


@pytest.fixture(scope="module")
def service_warp(tmp_path_factory):
    return _device_model(tmp_path_factory, "service_warp",
                         _extract(os.path.join(CSRC, "lbm_pair.cuh"), "struct PairShared",
                                  "__device__ __forceinline__ bool pair_ready",
                                  "__device__ __forceinline__ void pair_serve"))


@pytest.mark.parametrize("ranges", [(1, 1, 1), (2, 0, 3), (12, 12, 12)])
@pytest.mark.parametrize("polls", [0, 300])
def test_the_odd_step_is_ordered_after_every_group_it_needs(service_warp, ranges, polls):
    """The even tiles that any lane of the service warp polled are ordered
    before the compute warps' odd step, ready at once or after waiting; fewer
    and more groups than lanes."""
    p = subprocess.run([service_warp, *map(str, ranges), str(polls)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout + p.stderr


@pytest.fixture(scope="module")
def compute_warps(tmp_path_factory):
    pair = open(os.path.join(CSRC, "lbm_pair.cuh")).read()
    waits = pair[pair.index("// Compute warps: their even nodes"):pair.index("// Small domains:")]
    return _device_model(tmp_path_factory, "compute_warps",
                         waits + "\n" + _extract(os.path.join(CSRC, "lbm_kernels_fp64.cu"), "    k_list_two_fp64("))


@pytest.mark.parametrize("push", [0, 1])
@pytest.mark.parametrize("named,go", [(1, 1), (0, 1), (1, 0), (0, 0)])
def test_no_run_record_is_followed_whose_wait_ran_out(compute_warps, push, named, go):
    p = subprocess.run([compute_warps, str(push), str(named), str(go)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout + p.stderr
