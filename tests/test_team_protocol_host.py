"""The team PCG kernel (csrc/pcg_team.cu) on the CPU: its source, compiled for
the host, runs in an emulator of CTAs (tests/emu) that chooses the
interleaving.  Solves of the layouts that a small GPU test does not reach are
checked against the residual formed in double; the waits of the error and
restart paths are checked on the interleavings that a GPU takes once in a very
long time, where a wait that nothing ends is reported as a hang."""
import os
import re
import subprocess

import pytest

from artisynth_core_b200 import _lib as L

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EMU = os.path.join(ROOT, "tests", "emu")
CSRC = os.path.join(ROOT, "artisynth_core_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


def _without_function(src, head):
    """src without the function whose definition starts with `head`."""
    a = src.index(head)
    i = src.index("{", a)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        i += 1
        if depth == 0:
            return src[:a] + src[i:]


def kernel_source(path=os.path.join(CSRC, "pcg_team.cu")):
    """The planner and the kernel for the host: the helpers that are inline PTX
    come from the emulator, shared variables from the running CTA."""
    src = open(path).read()
    src = src[:src.index("static std::mutex g_team_mu;")] + "}  // namespace b200fem\n"
    for head in ("__device__ __forceinline__ void put_packet(", "__device__ __forceinline__ double get_packet(",
                 "__device__ __forceinline__ unsigned long long team_ns(", "__device__ __forceinline__ void row_barrier("):
        src = _without_function(src, head)
    src = src.replace("extern __shared__ __align__(16) unsigned char dyn[];", "unsigned char* const dyn = emu::dyn();")

    def shared(m):
        out = []
        for var in m.group(2).split(","):
            name, dims = re.match(r"\s*(\w+)((?:\[\w+\])*)", var).groups()
            t = m.group(1) + dims
            out.append(f"auto& {name} = emu::shared<{t}>(\"{name}\");")
        return " ".join(out)

    src = re.sub(r"__shared__ (\w+) ([^;]+);", shared, src)
    assert "__shared__" not in src and "asm" not in re.sub(r"//.*", "", src)
    return src


def build(tmp, path=None):
    with open(os.path.join(tmp, "team_kernel.inc"), "w") as f:
        f.write(kernel_source(path) if path else kernel_source())
    exe = os.path.join(tmp, "team_emu")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-U_FORTIFY_SOURCE", "-w", "-pthread", "-I", str(tmp), "-I", EMU, "-I", CSRC, "-I", CUDA_INC,
                        os.path.join(EMU, "team_emu.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


@pytest.fixture(scope="module")
def emu(tmp_path_factory):
    exe = build(str(tmp_path_factory.mktemp("emu")))

    def run(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0, (r.returncode, r.stderr)
        return dict(line.split(" ", 1) for line in r.stdout.splitlines())

    return run


SOLVES = {  # grids, stiffness, dil, fp32, CTAs, shared memory KB, variant, what the plan has to show
    "one_cta": ("4x3x3", "30", 0, 0, 1, 227, 0, {"sets": "1", "team": "1"}),
    "three_sets": ("9x6x6", "10", 0, 0, 1, 227, 0, {"sets": "3", "team": "1"}),
    "three_sets_fp32": ("9x6x6", "10", 0, 1, 1, 227, 0, {"sets": "3", "team": "1"}),
    "three_sets_nodal": ("31x5x2", "10", 1, 0, 1, 227, 0, {"sets": "3", "team": "1"}),
    "three_sets_nodal_fp32": ("31x5x2", "10", 1, 1, 1, 227, 0, {"sets": "3", "team": "1"}),
    "streamed_classic": ("9x6x6", "10", 0, 0, 1, 100, 1, {"sets": "3", "kept": "30", "streamed": "200"}),
    "streamed_pipelined": ("9x6x6", "10", 0, 0, 1, 100, 2, {"sets": "3", "kept": "30", "streamed": "200"}),
    "team_of_two": ("10x10x9", "10", 0, 1, 2, 227, 0, {"sets": "3", "team": "2"}),
    "nodal_team_streamed": ("8x8x8", "10", 1, 0, 4, 110, 0, {"sets": "1", "team": "4"}),
}


@pytest.mark.parametrize("name", list(SOLVES))
def test_solves(name, emu):
    grids, stiff, dil, fp32, ctas, kb, variant, shows = SOLVES[name]
    out = emu("solve", grids, stiff, 1e-9, dil, fp32, ctas, kb, variant)
    assert out["ended"] == "yes" and out["flag"] == "0" and out["converged"] == "1", out
    # the kernel accepts a true residual of at most tol; forming it again in another order moves it by rounding only
    assert float(out["residual"]) <= 1e-9 * (1 + 1e-3), out
    assert shows.items() <= out.items(), out


@pytest.mark.parametrize("warp", [0, 1, 7, 15])
def test_error_recorded_while_a_cta_starts(warp, emu):
    """The CTA's threads leave together or run together, whichever of its warps could see the error first."""
    out = emu("late_flag", warp)
    assert out["ended"] == "yes", out


@pytest.mark.parametrize("seed", [0, 3, 29, 47])
def test_restart_within_rounding_of_the_tolerance(seed, emu):
    """The verdict on the true residual is read by every warp before the restart writes its first code, and the restart
    iterates even where the square of the residual rounds to the threshold (seeds 3 and 47)."""
    out = emu("restart", seed)
    assert out["ended"] == "yes" and out["flag"] == "0" and out["converged"] == "1", out
    assert float(out["residual"]) <= 1e-12, out


def test_queueing_for_a_team_is_no_timeout(emu):
    """The first member of a team waits for the CTA that solves another model for 16 ms with a limit of 1 ms."""
    out = emu("queue")
    assert out["ended"] == "yes" and out["flag"] == "0" and out["converged"] == "1", out
    assert float(out["residual"]) <= 1e-8 * (1 + 1e-3) and int(out["clock_us"]) >= 10000, out


def test_lost_packets_of_a_complete_team_time_out(emu):
    out = emu("queue", "gone")
    assert out["ended"] == "yes" and out["flag"] == str(L.ERR_TIMEOUT), out


@pytest.mark.parametrize("seed", [0, 1, 2, 5])
@pytest.mark.parametrize("at", [0, 100000, -1])
def test_random_interleavings(seed, at, emu):
    """Three models on three CTAs, with and without an error recorded or found on the way: every thread ends, and the solve that
    follows is right."""
    out = emu("random", seed, at, seed % 3, seed // 3)
    assert out["ended"] == "yes", out
    if at < 0:
        assert out["flag"] == str(L.ERR_INVALID_ARG), out
    if at == 0:
        assert out["flag"] == "0" and float(out["residual"]) <= 1e-6 * (1 + 1e-3), out
    assert out["again"] == "yes" and out["again_flag"] == "0", out
    assert float(out["again_residual"]) <= 1e-6 * (1 + 1e-3), out


@pytest.mark.parametrize("variant", [0, 1, 2])
def test_error_recorded_while_a_warp_lags(variant, emu):
    """A poll that gives up after the last iteration does not take a slower warp out of the loop by another way."""
    out = emu("slow_warp", variant)
    assert out["ended"] == "yes" and out["team"] == "2" and out["flag"] != "0", out
