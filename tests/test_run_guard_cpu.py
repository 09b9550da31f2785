"""What a run gives back when it returns before its last host wait (cancelled,
an error): the library's own guard over a run, compiled against stand-ins for
the runtime calls it makes.  No device."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>

#include <string>

#include "dgpu_internal.h"

static std::string seen;                    // w: wait, a: pinned block taken, f: freed
static int held = 0;
extern "C" cudaError_t cudaStreamSynchronize(cudaStream_t) { seen += 'w'; return cudaSuccess; }
extern "C" cudaError_t cudaMallocHost(void **p, size_t n) { seen += 'a'; held++; *p = malloc(n); return cudaSuccess; }
extern "C" cudaError_t cudaFreeHost(void *p) { seen += 'f'; held--; free(p); return cudaSuccess; }
extern "C" cudaError_t cudaMalloc(void **, size_t) { return cudaErrorMemoryAllocation; }
extern "C" cudaError_t cudaFree(void *) { return cudaSuccess; }

// a run that stages n bytes and returns with or without its last host wait
static void run(HostArena &stage, dgpu_ctx *c, size_t n, bool finishes)
{
    RunGuard guard(c);
    if (!stage.take(n)) abort();
    if (!finishes) return;
    cudaStreamSynchronize(c->stream);
    guard.done = true;
    stage.reset();
}

int main()
{
    dgpu_ctx *c = new dgpu_ctx();
    run(c->stage, c, 1000, true);
    printf("%s\n", seen.c_str());
    seen.clear();
    run(c->stage, c, 1000, false);          // waits
    printf("%s\n", seen.c_str());
    for (int k = 0; k < 100; k++) run(c->stage, c, (size_t)300 << 10, false);
    printf("%d %zu\n", held, c->stage.cap);
    return 0;
}
"""


@pytest.mark.skipif(not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")),
                    reason="needs g++ and the CUDA headers")
def test_unfinished_runs_wait_and_give_the_staging_back(tmp_path):
    src = tmp_path / "guard.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "guard"
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(CUDA, "include"),
                           "-I", os.path.join(ROOT, "diffusecode_gb300", "csrc"), str(src), "-o", str(exe)])
    out = subprocess.check_output([str(exe)], text=True).split("\n")
    assert out[0] == "aw"                       # a finished run waits once
    assert out[1] == "w"                        # an unfinished one is waited for by the guard
    assert out[2] == "1 1048576"                # a hundred of them stay within the first block
