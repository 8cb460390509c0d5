"""The library's host code (plans, launches, waits, errors) on a machine without a GPU:
libbgp.so in a process of its own whose CUDA runtime is tests/fake_cudart.cpp, which runs
no kernel but notes launches, orders the legacy default stream and fails calls on request.
"""
import json
import os
import re
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# A process without torch (whose libraries would bring the real runtime): the binding
# module alone, with a placeholder for torch.
PRELUDE = r"""
import ctypes, importlib.util, json, sys, threading, types
fake = ctypes.CDLL(sys.argv[1])
fake.fake_count.restype = ctypes.c_longlong
fake.fake_stream.restype = ctypes.c_void_p
torch = types.ModuleType("torch"); torch._C = object(); sys.modules["torch"] = torch
spec = importlib.util.spec_from_file_location("binding", sys.argv[2])
L = importlib.util.module_from_spec(spec); spec.loader.exec_module(L)
lib = L.lib()
count = lambda what: fake.fake_count(what.encode())
def mallocs():
    n = fake.fake_mallocs(None, 0)
    a = (ctypes.c_size_t * n)()
    fake.fake_mallocs(a, n)
    return list(a)
def desc(N=16, ndim=2, kernel="none", beta2=10.0, beta3=0.0):
    return L.InstanceDesc(ndim, N, 2, L.KERNEL_CODES[kernel], 6.0, 2.0, 0.5, beta2, beta3, 0.0,
                          5.0 if kernel != "none" else 0.0, 0.0)
def plan(*descs):
    h = ctypes.c_void_p()
    rc = lib.bgp_plan_create((L.InstanceDesc * len(descs))(*descs), len(descs), ctypes.byref(h))
    return rc, h
def field(n):
    return (ctypes.c_double * (2 * n))()
def solve(h, n, points, stream=None, mixed=1, maxit=1, trials=4):
    p = L.SolverParams(maxit, trials, 4, 10, 0, 10, 0, 0, mixed, 1e-8, 1e-12, 0.1, 1.0, 0.1, 1e-3)
    f = [field(points) for _ in range(n)]
    P = (ctypes.c_void_p * n)(*[ctypes.addressof(x) for x in f])
    return lib.bgp_solve(h, P, P, ctypes.byref(p), (L.SolveResult * n)(), None, stream)
def apply(h, points, stream=None, n=1):
    f, g = [field(points) for _ in range(n)], [field(points) for _ in range(n)]
    P = lambda q: (ctypes.c_void_p * n)(*[ctypes.addressof(x) for x in q])
    return lib.bgp_apply_H_batch(h, n, (ctypes.c_int * n)(*range(n)), P(f), P(g), None, 2, None, stream)
out = {}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    nvcc = os.environ.get("NVCC", "nvcc")
    if shutil.which(nvcc) is None or shutil.which("g++") is None:
        pytest.skip("nvcc or g++ is not on PATH")
    d = tmp_path_factory.mktemp("fake_runtime")
    src, obj, so, vmap = os.path.join(ROOT, "tests", "fake_cudart.cpp"), d / "hooks.o", d / "libcudart.so.12", d / "v.map"
    vmap.write_text("libcudart.so.12 { global: cuda*; __cuda*; fake_*; local: *; };\n")
    home = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which(nvcc))))
    subprocess.run([nvcc, "-x", "cu", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O0", "-w",
                    "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "becgpp_b200", "csrc"), "-c", src, "-o", str(obj)],
                   check=True)
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-shared", "-fPIC", "-I", os.path.join(home, "include"), src, str(obj),
                    "-o", str(so), "-Wl,-soname,libcudart.so.12", f"-Wl,--version-script={vmap}"], check=True)

    def go(scenario):
        r = subprocess.run([sys.executable, "-c", PRELUDE + scenario + "\nprint(json.dumps(out))", str(so),
                            os.path.join(ROOT, "becgpp_b200", "_lib.py")], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr
        return json.loads(r.stdout.splitlines()[-1])
    return go


def test_a_mixed_solve_runs_to_its_end(run):
    got = run(r"""
rc, h = plan(desc())
out["rc"] = rc, solve(h, 1, 256), solve(h, 1, 256, stream=fake.fake_stream())
out["launches"] = count("k_sv_px")
lib.bgp_plan_destroy(h)
""")
    assert got["rc"] == [0, 0, 0] and got["launches"] > 0


def test_only_plan_creation_reads_the_shared_tables():
    """The maps of a device's tables grow under the creation lock; other threads' calls on
    other plans hold no lock, so they must not read them."""
    src = open(os.path.join(ROOT, "becgpp_b200", "csrc", "bgp_api.cu")).read()
    used, name = set(), None
    for line in src.splitlines():
        m = re.match(r"(?:template.*> *)?(?:int|void|bool|const \w+\*|long long|Sched) (\w+)\(", line)
        name = m.group(1) if m else name
        if re.search(r"(->|\.)(lf|lf32|tw)\b(\[|\.)", line):
            used.add(name)
    assert used == {"twiddles", "lf_table", "bgp_plan_create"}


@pytest.mark.parametrize("N,kernel", [(16, "none"), (24, "log"), (48, "none")])
def test_tables_of_a_failed_creation_are_complete_or_absent(run, N, kernel):
    """Whichever allocations of earlier creations failed, a mixed solve finds every line
    table, the FP32 ones too."""
    got = run(f"""
d = desc({N}, kernel="{kernel}")
rcs = []
for k in range(1, 40):
    fake.fake_fail_malloc(k)
    rc, h = plan(d)
    rcs.append(rc)
    if rc == 0: lib.bgp_plan_destroy(h)
fake.fake_fail_malloc(0)
rc, h = plan(d)
out.update(failed=sum(r != 0 for r in rcs), rc=[rc, solve(h, 1, {N * N})], null=count("null_table"), px=count("k_sv_px"))
""")
    assert got["failed"] >= 10 and got["rc"] == [0, 0] and got["px"] > 0
    assert got["null"] == 0


def test_memory_is_cleared_before_another_stream_uses_it(run):
    """The clearing of a plan's memory, and of the mixed solver's (allocated by its first
    solve), is over before anything runs on a stream the default stream does not order."""
    got = run(r"""
st = fake.fake_stream()
rc, h = plan(desc())
out["create"] = rc, apply(h, 256, st), count("unordered")
out["mixed"] = solve(h, 1, 256, st), count("unordered")
""")
    assert got == {"create": [0, 0, 0], "mixed": [0, 0]}


@pytest.mark.parametrize("N,beta3,step", [(384, 0.0, 1), (384, 0.0, 7), (256, 5.0, 9), (64, 0.0, 3)])
def test_a_timed_out_thomas_fermi_barrier_is_reported(run, N, beta3, step):
    """The status word of a step survives the steps enqueued after it, whichever team takes
    them (a grid at 384^2 and, with beta3 > 0, at 256^2; a cluster at 64^2, which reads the
    word that the cooperative seed may have set)."""
    got = run(f"""
rc, h = plan(desc({N}, kernel="log", beta3={beta3}))
n, info = (ctypes.c_double * {N * N})(), (ctypes.c_double * 5)()
tf = lambda: lib.bgp_tf_density(h, 0, 1, 0.0, 12, 0.3, ctypes.addressof(n), info, None)
out["fine"] = tf(), info[3]
fake.fake_tf_timeout({step})
out["timeout"] = tf(), lib.bgp_last_error().decode()
out["again"] = tf(), info[3]
""")
    assert got["fine"] == got["again"] == [0, 12.0]
    assert got["timeout"][0] == -4 and "timeout" in got["timeout"][1]


def test_mixed_solves_do_not_tune_the_relaunch_schedule(run):
    """Only FP64 solves are launches that yield; the timing of others says nothing about it."""
    got = run(r"""
rc, h = plan(desc(), desc(beta2=20.0))
def schedule():
    div, tuned, ms = ctypes.c_int(), ctypes.c_int(), (ctypes.c_float * 3)()
    assert lib.bgp_plan_schedule(h, ctypes.byref(div), ctypes.byref(tuned), ms) == 0
    return [div.value, tuned.value, list(ms)]
lib.bgp_plan_autotune(h, 1)
before = schedule()
out["mixed"] = [solve(h, 2, 256) for _ in range(4)], schedule() == before
out["fp64"] = [solve(h, 2, 256, mixed=0) for _ in range(3)], schedule()[1:]
""")
    assert got["mixed"] == [[0] * 4, True]
    assert got["fp64"] == [[0] * 3, [1, [1.0, 1.0, 1.0]]]


@pytest.mark.parametrize("clusters", [1, 0])
def test_thomas_fermi_without_room_for_a_cluster(run, clusters):
    """A device (or a partition of one) that cannot hold the cluster takes grid-wide steps."""
    got = run(f"""
fake.fake_clusters({clusters})
rc, h = plan(desc(64, kernel="log"))
n, info = (ctypes.c_double * 4096)(), (ctypes.c_double * 5)()
tf = lambda: lib.bgp_tf_density(h, 0, 1, 0.0, 5, 0.3, ctypes.addressof(n), info, None)
out["rc"] = tf(), tf()
out["steps"] = count("k_tf_iter_cluster"), count("k_tf_iter")
""")
    assert got == {"rc": [0, 0], "steps": [10, 0] if clusters else [0, 10]}


def test_a_failed_allocation_is_reported_once(run):
    """After a mixed solve, a plan or pinned memory that found no memory, other calls work."""
    got = run(r"""
rc, h = plan(desc())
fake.fake_fail_malloc(3)
out["solve"] = solve(h, 1, 256), apply(h, 256), solve(h, 1, 256), apply(h, 256)
fake.fake_fail_malloc(2)
out["plan"] = plan(desc(24))[0], apply(h, 256)
""")
    assert got["solve"] == [-3, 0, 0, 0]
    assert got["plan"] == [-3, 0]
    got = run(r"""
fake.fake_fail_host_alloc(1)                     # the device's block: the plan takes memory of its own
rc, h = plan(desc())
out["pinned"] = rc, apply(h, 256), lib.bgp_plan_destroy(h), count("live") >= 0
""")
    assert got["pinned"] == [0, 0, 0, True]


def test_a_line_search_of_no_trials_has_none_in_the_mixed_form(run):
    """linesearch_max = 0 stalls at the initial state: the FP64 solver's answer, not a solve
    whose launches each hold a trial."""
    got = run(r"""
rc, h = plan(desc())
out["rc"] = rc, solve(h, 1, 256, trials=0), solve(h, 1, 256, trials=-1), count("k_sv_trial")
out["one"] = solve(h, 1, 256, trials=1), count("k_sv_trial") > 0
""")
    assert got == {"rc": [0, 0, 0, 0], "one": [0, True]}
