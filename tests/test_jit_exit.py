"""A process that ends while a kernel instance is compiled on the background thread ends in order.

csrc/lyap_jit.cu is built as host code with a fake of the few CUDA runtime calls it makes (no device here), a launch asks for
work enough to start a compilation, and main returns while NVRTC is at it."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "lyapunovfractalwasm_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

MAIN = r"""
#include <cstdlib>
#include <cstring>
#include <thread>
#include <unistd.h>
#include <cuda_runtime.h>
#include "lyap_engine.h"
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void**, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorUnknown; }
}
static bool launched() {
    static lyap::LambdaArgs a;
    a.n_pixels = 1 << 30;
    a.width = 1 << 15;
    a.warmup = 90;
    a.iterations = 900;
    a.wu_wrap = a.acc_wrap = a.acc_word0 = 1;   // period 2: one word a region
    a.sel[0] = a.sel[1] = 0x44444444u;
    bool yes = true;
    const cudaError_t e = lyap::launch_lambda_spec(a, nullptr, nullptr, nullptr, 1, nullptr, 0, 2, 512, 0, 1, &yes);
    return e != cudaSuccess || yes;
}
// Once there is code, a launch tries to load it, and says that the fake driver cannot.
static void look() {
    launched();
    if (!*lyap::jit_last_note()) _exit(4);
}
static void at_the_end() { std::thread(look).join(); }
int main(int, char** argv) {
    std::atexit(at_the_end);
    if (launched()) return 3;   // the generic kernel's turn
    usleep(std::atoi(argv[1]) * 1000);
    return 0;
}
"""


def test_a_process_may_end_while_an_instance_is_compiled(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "include", "nvrtc.h")):
        pytest.skip("no CUDA headers")
    from lyapunovfractalwasm_b200 import build
    build.generate_jit_source()
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "ends")
    subprocess.run(["g++", "-std=c++20", "-O1", "-I", os.path.join(CUDA, "include"), "-I", CSRC, "-o", exe, str(tmp_path / "main.cpp"),
                    "-x", "c++", os.path.join(CSRC, "lyap_jit.cu"), "-ldl", "-lpthread"], check=True)
    env = dict(os.environ)
    env["LD_LIBRARY_PATH"] = os.path.join(CUDA, "lib64") + ":" + env.get("LD_LIBRARY_PATH", "")
    for ms in (500, 800):
        assert subprocess.run([exe, str(ms)], timeout=60, env=env).returncode == 0, ms   # 4: main's end did not wait for the compilation
