"""Build recipe: compiles the CUDA engine (sm_100a only) into lyapunovfractalwasm_b200/liblyap_b200.so.

nvcc cross-compiles without a GPU.  -fmad=false keeps nvcc from fusing a*b+c on its own: the exact
kernels fuse only where an fma is written out (see csrc/lyap_math.h).
"""
import os
import subprocess
import sys

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(HERE, "csrc")
LIB = os.path.join(HERE, "liblyap_b200.so")

NVCC_FLAGS = [
    "-std=c++20", "-O3", "-lineinfo",
    "-gencode", "arch=compute_100a,code=sm_100a",
    "-fmad=false",
    "-Xcompiler", "-fPIC,-ffp-contract=off,-Wall",
]
OBJ_DIR = os.path.join(HERE, "build")

# Lambda-kernel instances compiled ahead of time and embedded in the library (csrc/lyap_prebuilt.cu):
# (sequence, 'C' selects a third parameter, warm-up steps) of the benchmark frames ...
PREBUILT_SEQUENCES = [("AB", False, 100), ("AABAB", False, 200), ("BBBBBBAAAAAA", False, 500), ("ABC", True, 300),
                      ("ABB", False, 300)]
# ... in the shapes the launchers ask for:
# (kind: 0 exact / 1 fast fp64 / 2 fast fp32 / 3 fast fp64 on the exact orbit, pixels per thread, threads)
PREBUILT_SHAPES = [(0, 2, 512), (1, 2, 128), (2, 2, 128), (3, 2, 128)]
NVRTC_OPTIONS = ["--gpu-architecture=sm_100a", "--fmad=false", "--std=c++17", "-lineinfo"]   # as csrc/lyap_jit.cu passes them


def _newer(target, sources):
    if not os.path.exists(target):
        return True
    t = os.path.getmtime(target)
    return any(os.path.getmtime(s) > t for s in sources)


HEADERS = ["lyap_exact_kernel.cuh", "lyap_kernels_fast.cuh", "lyap_engine.h", "lyap_args.h", "lyap_math.h", "lyap_tables.h"]
UNITS = ["lyap_abi.cu", "lyap_kernels.cu", "lyap_jit.cu", "lyap_multi.cu", "lyap_prebuilt.cu"]


def lib_sources():
    names = UNITS + HEADERS
    return [os.path.join(CSRC, n) for n in names] + [os.path.join(ROOT, "include", "lyap_b200.h")]


JIT_INC = os.path.join(CSRC, "lyap_jit_source.inc")
JIT_FILES = ["lyap_exact_kernel.cuh", "lyap_kernels_fast.cuh", "lyap_args.h", "lyap_math.h", "lyap_tables.h"]


def generate_jit_source():
    """Embed the exact kernel's sources as text for the run-time specialiser (csrc/lyap_jit.cu)."""
    out = ["// GENERATED by build.py from %s -- do not edit." % ", ".join(JIT_FILES)]
    for name in JIT_FILES:
        text = open(os.path.join(CSRC, name)).read()
        var = "kSrc_" + name.replace(".", "_")
        out.append("static const char %s[] =" % var)
        size = -(-len(text) // -(-len(text) // 8000))   # string literals are concatenated; small pieces of one size
        for i in range(0, len(text), size):
            out.append('R"LYAPSRC(' + text[i:i + size] + ')LYAPSRC"')
        out.append(";")
    new = "\n".join(out) + "\n"
    if not os.path.exists(JIT_INC) or open(JIT_INC).read() != new:
        with open(JIT_INC, "w") as f:
            f.write(new)


def sequence_patterns(sequence, use_c, warmup):
    """(KG, warm-up patterns, accumulation patterns) of a long run of `sequence`: the smallest number KG of two-step
    groups after which the parameter choices repeat, and the 2-bit codes (0 = A, 1 = B, 2 = C) of one such period from
    step 0 and from step `warmup` -- what sequence_group_period (csrc/lyap_jit.cu) finds for the same run."""
    def code(i):
        ch = sequence[i % len(sequence)]
        return 0 if ch == "A" else (2 if (use_c and ch == "C") else 1)
    for kg in range(1, 17):
        if all(code(i) == code(i + 2 * kg) for i in range(4 * len(sequence))):
            pats = lambda first: sum(code(first + i) << (2 * i) for i in range(2 * kg))
            return kg, pats(0), pats(warmup)
    raise ValueError("no group period up to 16 for " + sequence)


def nvrtc_compile(sources, options):
    """One program (the two kernel headers) through NVRTC -> cubin bytes.  Needs no GPU."""
    import ctypes
    lib = None
    for name in ("libnvrtc.so.12", "/usr/local/cuda/lib64/libnvrtc.so.12", "libnvrtc.so"):
        try:
            lib = ctypes.CDLL(name)
            break
        except OSError:
            pass
    if lib is None:
        raise RuntimeError("libnvrtc (part of the CUDA toolkit) not found: it compiles the embedded kernel instances")
    names = list(sources)
    hs = (ctypes.c_char_p * len(names))(*[sources[n].encode() for n in names])
    hn = (ctypes.c_char_p * len(names))(*[n.encode() for n in names])
    main = b'#include "lyap_exact_kernel.cuh"\n#include "lyap_kernels_fast.cuh"\n'
    prog = ctypes.c_void_p()
    if lib.nvrtcCreateProgram(ctypes.byref(prog), main, b"lyap_spec.cu", len(names), hs, hn) != 0:
        raise RuntimeError("nvrtcCreateProgram failed")
    opts = (ctypes.c_char_p * len(options))(*[o.encode() for o in options])
    rc = lib.nvrtcCompileProgram(prog, len(options), opts)
    if rc != 0:
        n = ctypes.c_size_t()
        lib.nvrtcGetProgramLogSize(prog, ctypes.byref(n))
        log = ctypes.create_string_buffer(n.value)
        lib.nvrtcGetProgramLog(prog, log)
        raise RuntimeError("NVRTC: " + log.value.decode(errors="replace")[-2000:])
    n = ctypes.c_size_t()
    lib.nvrtcGetCUBINSize(prog, ctypes.byref(n))
    cubin = ctypes.create_string_buffer(n.value)
    lib.nvrtcGetCUBIN(prog, cubin)
    lib.nvrtcDestroyProgram(ctypes.byref(prog))
    return cubin.raw


PREBUILT_TABLE = os.path.join(CSRC, "lyap_prebuilt_table.inc")
PREBUILT_BLOB = os.path.join(CSRC, "lyap_prebuilt_blob.bin")
PREBUILT_STUB = os.path.join(CSRC, "lyap_prebuilt_blob.S")


def generate_prebuilt():
    """Compiles the embedded instances (same source text and options as a run-time instance) and writes the three
    generated files lyap_prebuilt.cu builds on: the table of instances, their device code back to back, and the
    assembler stub that places that code in the library's read-only data."""
    import hashlib
    from concurrent.futures import ThreadPoolExecutor
    sources = {n: open(os.path.join(CSRC, n)).read() for n in JIT_FILES}
    jobs = []
    for seq, use_c, warmup in PREBUILT_SEQUENCES:
        kg, wu, acc = sequence_patterns(seq, use_c, warmup)
        for kind, ppt, threads in PREBUILT_SHAPES:
            kind_opt = ["-DLYAP_SPEC_EXACT=1", "-DLYAP_SPEC_FAST=FusedF64", "-DLYAP_SPEC_FAST=FusedF32",
                        "-DLYAP_SPEC_FAST=OrbitF64"][kind]
            opts = NVRTC_OPTIONS + ["-DLYAP_SPEC_THREADS=%d" % threads, kind_opt, "-DLYAP_SPEC_P=%d" % ppt,
                                    "-DLYAP_SPEC_KG=%d" % kg, "-DLYAP_SPEC_WU_PATS=0x%xull" % wu,
                                    "-DLYAP_SPEC_ACC_PATS=0x%xull" % acc]
            jobs.append((kind, ppt, threads, kg, wu, acc, seq, opts))
    stamp = hashlib.sha256(repr((sorted(sources.items()), [j[:7] + (j[7],) for j in jobs])).encode()).hexdigest()
    head = "// GENERATED by build.py (generate_prebuilt); inputs %s\n" % stamp
    if all(os.path.exists(f) for f in (PREBUILT_TABLE, PREBUILT_BLOB, PREBUILT_STUB)) and \
            open(PREBUILT_TABLE).readline() == head:
        return
    with ThreadPoolExecutor(max_workers=os.cpu_count() or 4) as pool:
        cubins = list(pool.map(lambda j: nvrtc_compile(sources, j[7]), jobs))
    rows, blob = [], b""
    for (kind, ppt, threads, kg, wu, acc, seq, _o), cubin in zip(jobs, cubins):
        blob += b"\0" * (-len(blob) % 16)
        rows.append('    {%d, %d, %d, %d, 0x%xull, 0x%xull, %d, %d, "%s"},' % (kind, ppt, threads, kg, wu, acc, len(blob), len(cubin), seq))
        blob += cubin
    with open(PREBUILT_BLOB, "wb") as f:
        f.write(blob)
    with open(PREBUILT_STUB, "w") as f:
        f.write("// GENERATED by build.py: the embedded kernel instances as read-only data\n"
                '    .section .rodata\n    .balign 16\n    .global lyap_prebuilt_blob\nlyap_prebuilt_blob:\n'
                '    .incbin "%s"\n    .section .note.GNU-stack,"",@progbits\n' % PREBUILT_BLOB)
    with open(PREBUILT_TABLE, "w") as f:
        f.write(head + "\n".join(rows) + "\n")


def build_library(force=False, verbose=False):
    """Compiles every translation unit to an object (in parallel) and links liblyap_b200.so."""
    from concurrent.futures import ThreadPoolExecutor
    generate_jit_source()
    generate_prebuilt()
    srcs = lib_sources() + [PREBUILT_TABLE, PREBUILT_BLOB]
    if not force and not _newer(LIB, srcs):
        return LIB
    os.makedirs(OBJ_DIR, exist_ok=True)
    extra = ["-Xptxas", "-v"] if verbose else []
    jobs = [(os.path.join(CSRC, u), os.path.join(OBJ_DIR, u[:-3] + ".o"), []) for u in UNITS]

    def compile_one(job):
        src, obj, defs = job
        r = subprocess.run(["nvcc"] + NVCC_FLAGS + extra + defs + ["-c", "-o", obj, src], capture_output=True, text=True)
        return job, r

    with ThreadPoolExecutor(max_workers=min(len(jobs), os.cpu_count() or 4)) as pool:
        results = list(pool.map(compile_one, jobs))
    for (src, _obj, defs), r in results:
        if verbose or r.returncode != 0:
            sys.stderr.write("== %s %s\n%s%s" % (os.path.basename(src), " ".join(defs), r.stdout, r.stderr))
        if r.returncode != 0:
            raise RuntimeError("nvcc failed on " + src)
    blob_obj = os.path.join(OBJ_DIR, "lyap_prebuilt_blob.o")
    subprocess.run(["gcc", "-c", "-o", blob_obj, PREBUILT_STUB], check=True)
    subprocess.run(["nvcc", "-shared", "-cudart", "shared", "-gencode", "arch=compute_100a,code=sm_100a",
                    "-o", LIB + ".tmp"] + [obj for _s, obj, _d in jobs] + [blob_obj, "-ldl"], check=True)
    os.replace(LIB + ".tmp", LIB)     # never leave a half-written library where a loader could find it
    return LIB


CLI = os.path.join(HERE, "lyap_cli")


def build_cli(force=False):
    """The C++23 command-line driver (host code only; links the engine library)."""
    src = os.path.join(CSRC, "lyap_cli.cpp")
    if not force and not _newer(CLI, [src, os.path.join(ROOT, "include", "lyap_b200.h"), LIB]):
        return CLI
    subprocess.run(["g++", "-std=c++23", "-O2", "-Wall", "-o", CLI, src, "-L", HERE, "-llyap_b200",
                    "-Wl,-rpath,$ORIGIN"], check=True)
    return CLI


def build_oracle():
    """Compile the CPU checkers (test infrastructure).  Uses the reference sources only where present."""
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle")], check=True)


if __name__ == "__main__":
    build_library(force="--force" in sys.argv, verbose="-v" in sys.argv)
    build_cli(force="--force" in sys.argv)
    build_oracle()
    print(LIB)
