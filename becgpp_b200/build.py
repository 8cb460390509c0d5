"""Build libbgp.so in-tree for sm_100a.

One translation unit per compiled grid size (N, M) keeps every kernel small
enough for ptxas and lets the sizes compile in parallel; a generated header
lists the sizes for the host dispatcher. Objects are rebuilt only when a
source or header is newer.

    python -m becgpp_b200.build [-j JOBS] [--force] [--profile]

--profile builds a second library, libbgp_prof.so, from the same sources with
the phase profiler compiled in (-DBGP_PROF): thread 0 of every team's first CTA
accumulates, per kind of phase, the time spent working, reducing, waiting at
the team barrier and gathering the reduced values. Select it at run time with
BECGPP_B200_LIB=<path>; `python bench.py --case phases` does so and prints the
breakdown.
"""
import argparse
import concurrent.futures as cf
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "csrc")
BUILD = os.path.join(os.path.dirname(HERE), "_build", "bgp")
GEN = os.path.join(BUILD, "gen")
LIB = os.path.join(HERE, "libbgp.so")
PROF_LIB = os.path.join(HERE, "libbgp_prof.so")

# grid sizes compiled into the solver: N per axis, M = 2N with a long-range kernel
SIZES_N = (16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)
MAX_N_WITH_KERNEL = 384
# two-size kernels for batches that mix grids (sweeps over 128^2 and 256^2)
COMBOS = ((128, 0, 256, 0),)

# stream-pass candidates of the autotuner: lines per tile and factorization variants
# of the line transform (csrc/bgp_lfft.cuh)
STREAM_LINES = (2, 4, 8)
PAD_LINES = (4, 8)        # the padded, strided passes
VARIANTS = (0, 1)
SOLVER_SMALL = 4          # lines per tile of the solver's small configuration (kSvSmall)


NVCC = os.environ.get("NVCC", "nvcc")
ARCH = ["-gencode", "arch=compute_100a,code=sm_100a"]
FLAGS = ["-std=c++17", "-O3", "-lineinfo", "-Xcompiler", "-fPIC", "-Xcompiler", "-O2"]


def pairs():
    out = []
    for n in SIZES_N:
        out.append((n, 0))
        if n <= MAX_N_WITH_KERNEL:
            out.append((n, 2 * n))
    return out


def _write_if_changed(path, text):
    if os.path.isfile(path) and open(path).read() == text:
        return
    with open(path, "w") as f:
        f.write(text)


def generate():
    os.makedirs(GEN, exist_ok=True)
    units = []
    hdr = ["// generated by becgpp_b200/build.py: compiled grid sizes", "#pragma once",
           "namespace bgp { struct SKernel; }"]
    hdr.append("#define BGP_FOR_SIZES(X) " + " ".join(f"X({n}, {m})" for n, m in pairs()))
    hdr.append("#define BGP_FOR_COMBOS(X) " + " ".join(f"X({a}, {b}, {c}, {d})" for a, b, c, d in COMBOS))
    hdr.append("#define BGP_FOR_TABLE_LENGTHS(X) "
               + " ".join(f"X({m})" for m in sorted({m for _, m in pairs() if m})))
    # each persistent kernel per grid dimension (BGP_NDIM)
    for dim in (2, 3):
        pre = f"#define BGP_NDIM {dim}\n"
        for n, m in pairs():
            name = f"{n}_{m}_d{dim}"
            hdr.append(f'extern "C" void* bgp_kptr_{name}();')
            src = (pre + f'#include "bgp_kernel.cuh"\n'
                   f"template __global__ void bgp::bgp_kernel_t<{n}, {m}>(bgp::Launch);\n"
                   f'extern "C" void* bgp_kptr_{name}() {{ return (void*)&bgp::bgp_kernel_t<{n}, {m}>; }}\n')
            path = os.path.join(GEN, f"k_{name}.cu")
            _write_if_changed(path, src)
            units.append(path)
        if dim != 2:
            continue   # the two-size kernels serve 2D batches
        for a, b, c, d in COMBOS:
            name = f"{a}_{b}_{c}_{d}_d{dim}"
            hdr.append(f'extern "C" void* bgp_kptr2_{name}();')
            src = (pre + f'#include "bgp_kernel.cuh"\n'
                   f"template __global__ void bgp::bgp_kernel_t2<{a}, {b}, {c}, {d}>(bgp::Launch);\n"
                   f'extern "C" void* bgp_kptr2_{name}() '
                   f"{{ return (void*)&bgp::bgp_kernel_t2<{a}, {b}, {c}, {d}>; }}\n")
            path = os.path.join(GEN, f"k2_{name}.cu")
            _write_if_changed(path, src)
            units.append(path)
    # stream passes (standalone and batched H psi): per line length N the axis passes,
    # and per padded length M = 2N the convolution's, in every (lines per tile,
    # factorization) candidate of the autotuner, for one instance and for a batch
    def stream_unit(path, include, groups):
        lines = [f'#include "{include}"']
        for fn, kern, length, widths, kinds in groups:
            cases = []
            for ln in widths:
                for v in VARIANTS:
                    for k in kinds:
                        for nb in ("1", "bgp::kStreamBatch"):
                            if k is None and nb != "1":
                                continue
                            inst = f"bgp::{kern}<{length}, {ln}, {v}, {k}, {nb}>"
                            if k is None:          # the energy sums: all axes, one instance
                                inst = f"bgp::{kern}<{length}, {ln}, {v}>"
                            lines.append(f"template __global__ void {inst}(const __grid_constant__ bgp::SLaunchT<{nb}>);")
                            cases.append(f"  if (c == {ln} && v == {v} && k == {k or 0} && batch == {int(nb != '1')}) {{\n"
                                         f"    constexpr int th = bgp::s_threads({length}, {ln}, {v});\n"
                                         f"    constexpr size_t sm = bgp::s_smem({length}, {ln}, {v});\n"
                                         f"    static const bgp::SKernel e{{(void*)&{inst}, th, sm, bgp::s_min_blocks({length}, {ln}, {v})}};\n"
                                         f"    return &e;\n  }}")
            lines.append(f'extern "C" const bgp::SKernel* {fn}(int c, int v, int k, int batch) {{')
            lines += cases
            lines.append("  return nullptr;\n}")
            hdr.append(f'extern "C" const bgp::SKernel* {fn}(int c, int v, int k, int batch);')
        _write_if_changed(path, "\n".join(lines) + "\n")
        units.append(path)

        hdr.append("#define BGP_FOR_LINE_LENGTHS(X) "
               + " ".join(f"X({n})" for n in sorted({n for n, _ in pairs()} | {m for _, m in pairs() if m})))
    hdr.append("#define BGP_FOR_STREAM_N(X) " + " ".join(f"X({n})" for n in SIZES_N))
    hdr.append("#define BGP_FOR_STREAM_M(X) " + " ".join(f"X({2 * n})" for n in SIZES_N if n <= MAX_N_WITH_KERNEL))
    for n in SIZES_N:
        stream_unit(os.path.join(GEN, f"s_{n}.cu"), "bgp_stream.cuh",
                    [(f"bgp_sptr_{n}", "k_stream_h", n, STREAM_LINES, (0, 1, 2)),
                     (f"bgp_septr_{n}", "k_stream_energy", n, PAD_LINES, (None,))])
        if n <= MAX_N_WITH_KERNEL:
            m = 2 * n
            stream_unit(os.path.join(GEN, f"s_conv_{m}.cu"), "bgp_stream.cuh",
                        [(f"bgp_srptr_{m}", "k_stream_real", n, STREAM_LINES, (0, 1)),
                         (f"bgp_spptr_{m}", "k_stream_pad", m, PAD_LINES, (0, 1, 2))])
    # solver passes, three configurations per size (sv_step): tiles of 4 lines with the
    # most threads per line, of 4 lines with fewer, and of 8 lines; where two factorizations
    # coincide the first is used for both
    def solver_unit(path, fn, entries):
        lines, cases, seen = ['#include "bgp_solve.cuh"'], [], set()
        for cfg in (0, 1, 2):
            c = 8 if cfg == 2 else SOLVER_SMALL
            for k, (kern, L, mode) in enumerate(entries):
                pow2 = L & (L - 1) == 0
                v = (2, 1 if pow2 else 2, 0 if not pow2 or fn.startswith("bgp_svc") else 1)[cfg]
                args = [str(L), str(c), str(v)] + ([str(mode)] if mode is not None else [])
                inst = f"bgp::{kern}<{', '.join(args)}>"
                if inst not in seen:
                    seen.add(inst)
                    lines.append(f"template __global__ void {inst}(const __grid_constant__ bgp::SvLaunch);")
                low = f"(sm < {8 * 1024} ? {8 * 1024} : sm)" if kern == "k_sv_hx" else "sm"
                cases.append(f"  if (cfg == {cfg} && k == {k}) {{\n"
                             f"    constexpr int th = bgp::s_threads({L}, {c}, {v});\n"
                             f"    constexpr size_t sm = bgp::s_smem({L}, {c}, {v});\n"
                             f"    static const bgp::SKernel e{{(void*)&{inst}, th, {low}, "
                             f"bgp::{'s_min_blocks' if kern == 'k_sv_pad' else 'sv_blocks'}({L}, {c}, {v})}};\n"
                             f"    return &e;\n  }}")
        lines.append(f'extern "C" const bgp::SKernel* {fn}(int cfg, int k) {{')
        lines += cases
        lines.append("  return nullptr;\n}")
        hdr.append(f'extern "C" const bgp::SKernel* {fn}(int cfg, int k);')
        _write_if_changed(path, "\n".join(lines) + "\n")
        units.append(path)

    for n in SIZES_N:
        solver_unit(os.path.join(GEN, f"sv_{n}.cu"), f"bgp_svptr_{n}",
                    [("k_sv_trial", n, None), ("k_sv_hy", n, None), ("k_sv_hx", n, None), ("k_sv_p", n, 0),
                     ("k_sv_p", n, 1), ("k_sv_p", n, 2), ("k_sv_px", n, None)])
        if n <= MAX_N_WITH_KERNEL:
            m = 2 * n
            solver_unit(os.path.join(GEN, f"sv_conv_{m}.cu"), f"bgp_svcptr_{m}",
                        [("k_sv_real", n, 0), ("k_sv_real", n, 1), ("k_sv_pad", m, 0), ("k_sv_pad", m, 1),
                         ("k_sv_pad", m, 2)])
    _write_if_changed(os.path.join(GEN, "bgp_sizes_gen.h"), "\n".join(hdr) + "\n")
    return units


# headers the persistent solver kernels include (the generated per-size units);
# the host units (bgp_api.cu, bgp_noalloc.cu, bgp_diag.cu, bgp_vortex.cu) depend on every header
KERNEL_HEADERS = ("bgp_kernel.cuh", "bgp_programs.cuh", "bgp_passes.cuh", "bgp_device.cuh", "bgp_fft.cuh",
                  "bgp_common.cuh")


def _deps(src):
    # (the generated unit itself carries its instantiations, so build.py is no dependency)
    if os.path.basename(src).startswith(("k_", "k2_")):
        return [os.path.join(CSRC, f) for f in KERNEL_HEADERS]
    if os.path.basename(src).startswith("sv_"):
        return [os.path.join(CSRC, f) for f in KERNEL_HEADERS + ("bgp_solve.cuh", "bgp_stream.cuh", "bgp_lfft.cuh")]
    if os.path.basename(src).startswith("s_"):
        return [os.path.join(CSRC, f) for f in ("bgp_stream.cuh", "bgp_lfft.cuh", "bgp_device.cuh", "bgp_fft.cuh",
                                                "bgp_common.cuh")]
    return [os.path.join(CSRC, f) for f in os.listdir(CSRC) if f.endswith((".cuh", ".cu", ".h"))] + [
        os.path.join(os.path.dirname(HERE), "include", "bgp.h"), os.path.abspath(__file__)]


def _compile(src, obj, force):
    newest = max(os.path.getmtime(p) for p in _deps(src) + [src])
    if not force and os.path.isfile(obj) and os.path.getmtime(obj) >= newest:
        return obj, None
    cmd = [NVCC, *ARCH, *FLAGS, "-I", CSRC, "-I", GEN, "-c", src, "-o", obj]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if r.returncode != 0:
        return obj, f"{' '.join(cmd)}\n{r.stdout}\n{r.stderr}"
    return obj, None


def build(jobs=None, force=False, verbose=True):
    units = generate()
    units.append(os.path.join(CSRC, "bgp_api.cu"))
    units.append(os.path.join(CSRC, "bgp_noalloc.cu"))
    units.append(os.path.join(CSRC, "bgp_diag.cu"))
    units.append(os.path.join(CSRC, "bgp_vortex.cu"))
    os.makedirs(BUILD, exist_ok=True)
    objs = [os.path.join(BUILD, os.path.splitext(os.path.basename(u))[0] + ".o") for u in units]
    jobs = jobs or max(1, os.cpu_count() or 1)
    errors = []
    with cf.ThreadPoolExecutor(jobs) as ex:
        futs = [ex.submit(_compile, u, o, force) for u, o in zip(units, objs)]
        for f in cf.as_completed(futs):
            obj, err = f.result()
            if err:
                errors.append(err)
            elif verbose:
                print(f"[build] {os.path.basename(obj)}", flush=True)
    if errors:
        raise RuntimeError("nvcc failed:\n" + "\n".join(errors))
    newest = max(os.path.getmtime(o) for o in objs)
    if force or not os.path.isfile(LIB) or os.path.getmtime(LIB) < newest:
        cmd = [NVCC, *ARCH, "-shared", "-o", LIB, *objs, "-lcudart"]
        r = subprocess.run(cmd, capture_output=True, text=True)
        if r.returncode != 0:
            raise RuntimeError(f"link failed:\n{r.stdout}\n{r.stderr}")
    if verbose:
        print(f"[build] {LIB}", flush=True)
    return LIB


def build_profiler(jobs=None, force=False, verbose=True, sizes=None):
    """libbgp_prof.so: the same library with the phase profiler compiled in
    (optionally only the grid sizes N in `sizes`)."""
    global BUILD, GEN, LIB, FLAGS, SIZES_N
    saved = BUILD, GEN, LIB, FLAGS, SIZES_N
    BUILD = os.path.join(os.path.dirname(HERE), "_build", "bgp_prof")
    GEN = os.path.join(BUILD, "gen")
    LIB = PROF_LIB
    FLAGS = FLAGS + ["-DBGP_PROF"]
    if sizes:
        SIZES_N = tuple(sizes)
    try:
        return build(jobs, force, verbose)
    finally:
        BUILD, GEN, LIB, FLAGS, SIZES_N = saved


if __name__ == "__main__":
    ap = argparse.ArgumentParser()
    ap.add_argument("-j", "--jobs", type=int, default=None)
    ap.add_argument("--force", action="store_true")
    ap.add_argument("--profile", action="store_true", help="build libbgp_prof.so (phase profiler)")
    ap.add_argument("--sizes", default=None, help="--profile: comma-separated grid sizes N to compile")
    a = ap.parse_args()
    try:
        if a.profile:
            build_profiler(a.jobs, a.force, sizes=[int(x) for x in a.sizes.split(",")] if a.sizes else None)
        else:
            build(a.jobs, a.force)
    except RuntimeError as e:
        print(e, file=sys.stderr)
        sys.exit(1)
