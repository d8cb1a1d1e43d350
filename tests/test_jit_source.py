"""The run-time specialised kernel's source compiles for sm_100a without a GPU (NVRTC runs on the CPU).

The library embeds csrc/lyap_exact_kernel.cuh and its three headers as text and hands them to NVRTC with the
sequence's group patterns as macros (csrc/lyap_jit.cu); this test does the same through the Python NVRTC binding."""
import os

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lyapunovfractalwasm_b200", "csrc")


def test_specialised_kernel_source_compiles_for_sm_100a():
    try:
        from cuda.bindings import nvrtc
    except ImportError:
        nvrtc = pytest.importorskip("cuda.nvrtc")
    from lyapunovfractalwasm_b200 import build
    read = lambda n: open(os.path.join(CSRC, n)).read().encode()
    names = [b"lyap_exact_kernel.cuh", b"lyap_kernels_fast.cuh", b"lyap_args.h", b"lyap_math.h", b"lyap_tables.h"]
    main = b'#include "lyap_exact_kernel.cuh"\n#include "lyap_kernels_fast.cuh"\n'
    # "AABAB": group patterns AA BA BA AB AB for both regions (warm-up 200 is a whole number of periods)
    common = [b"--gpu-architecture=sm_100a", b"--fmad=false", b"--std=c++17", b"-DLYAP_SPEC_KG=5",
              b"-DLYAP_SPEC_WU_PATS=0x44110ull", b"-DLYAP_SPEC_ACC_PATS=0x44110ull"]
    kinds = [b"-DLYAP_SPEC_EXACT=1", b"-DLYAP_SPEC_FAST=FusedF64", b"-DLYAP_SPEC_FAST=FusedF32", b"-DLYAP_SPEC_FAST=OrbitF64"]
    for which, pixels, threads in build.PREBUILT_SHAPES:   # the shapes the launchers ask for
        symbol = b"k_lambda_exact_spec" if which == 0 else b"k_lambda_fast_spec"
        kind = [kinds[which], b"-DLYAP_SPEC_THREADS=%d" % threads, b"-DLYAP_SPEC_P=%d" % pixels]
        err, prog = nvrtc.nvrtcCreateProgram(main, b"spec.cu", len(names), [read(n.decode()) for n in names], names)
        assert err == nvrtc.nvrtcResult.NVRTC_SUCCESS
        opts = common + kind
        (err,) = nvrtc.nvrtcCompileProgram(prog, len(opts), opts)
        _, n = nvrtc.nvrtcGetProgramLogSize(prog)
        log = b" " * n
        nvrtc.nvrtcGetProgramLog(prog, log)
        assert err == nvrtc.nvrtcResult.NVRTC_SUCCESS, log.decode(errors="replace")[:3000]
        _, size = nvrtc.nvrtcGetCUBINSize(prog)
        cubin = b" " * size
        nvrtc.nvrtcGetCUBIN(prog, cubin)
        assert size > 10000 and symbol in cubin, kind      # the instance's kernel is really in there
        assert b"error" not in log.lower()


def test_embedded_source_is_current():
    """lyap_jit_source.inc (generated by build.py) holds exactly the files this test compiled."""
    from lyapunovfractalwasm_b200 import build
    build.generate_jit_source()
    inc = open(build.JIT_INC).read()
    for name in build.JIT_FILES:
        text = open(os.path.join(CSRC, name)).read()
        assert text[:200] in inc and text[-200:] in inc, name


def test_embedded_instances_are_keyed_as_the_library_keys_its_launches():
    """build.py embeds one instance per benchmark sequence under the key (groups, warm-up patterns, accumulation
    patterns) it computes in Python; a launch looks instances up under the key the library computes from the packed
    selectors (lyap_group_patterns).  Both must agree, or the embedded code would never run.  Also: every row of the
    generated table carries one of those keys, and the blob holds a cubin (ELF) at every offset."""
    import lyapunovfractalwasm_b200 as L
    from lyapunovfractalwasm_b200 import build
    build.generate_prebuilt()
    keys = set()
    for seq, use_c, warmup in build.PREBUILT_SEQUENCES:
        want = build.sequence_patterns(seq, use_c, warmup)
        p = L.make_params(width=64, height=64, sequence=seq, iterations=4000, warmup=warmup, c=3.7 if use_c else None)
        assert L.group_patterns(p) == want, seq
        keys.add(want)
    # other sequences with the same patterns share the instance; a different warm-up phase does not
    assert L.group_patterns(L.make_params(sequence="ABABABAB", iterations=500, warmup=100)) == build.sequence_patterns("AB", False, 100)
    assert L.group_patterns(L.make_params(sequence="AB", iterations=500, warmup=101))[2] != build.sequence_patterns("AB", False, 100)[2]
    assert L.group_patterns(L.make_params(sequence="ABBABAABBBABAABABBBAABABAABBBABBAAA", iterations=500, warmup=10))[0] == 0
    blob = open(build.PREBUILT_BLOB, "rb").read()
    rows = [l for l in open(build.PREBUILT_TABLE) if l.strip().startswith("{")]
    assert len(rows) == len(build.PREBUILT_SEQUENCES) * len(build.PREBUILT_SHAPES)
    for line in rows:
        f = [x.strip() for x in line.strip().strip("{},").split(",")]
        kg, wu, acc, off, size = int(f[3]), int(f[4].rstrip("ul"), 16), int(f[5].rstrip("ul"), 16), int(f[6]), int(f[7])
        assert (kg, wu, acc) in keys
        assert blob[off:off + 4] == b"\x7fELF" and off + size <= len(blob)
