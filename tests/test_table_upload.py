"""The upload of constant tables (csrc/bbdg_upload.cuh), compiled on the host against a recording
stand-in for the CUDA runtime: the allocation and the copy happen on the table's own device
whichever one the caller has current, outside any capture's restrictions, and the copy is waited
for before the pointer is handed out."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include "bbdg_upload.cuh"
static int current = 1;                       // the caller works on device 1
static bool relaxed = false, pending = false;
static const char* fail_at = "";
static bool fails(const char* what) { return std::strcmp(fail_at, what) == 0; }
static void say(const char* what) { std::printf("%s dev=%d relaxed=%d\n", what, current, relaxed); }
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { if (d == 7) return cudaErrorInvalidDevice; current = d; return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
  const bool was = relaxed;
  relaxed = *m == cudaStreamCaptureModeRelaxed;
  *m = was ? cudaStreamCaptureModeRelaxed : cudaStreamCaptureModeGlobal;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
  say("malloc");
  if (fails("malloc")) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) { say("free"); std::free(p); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  *s = (cudaStream_t)8;
  return f == cudaStreamNonBlocking ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
static void* to; static const void* from; static size_t count;
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  say("copy");
  if (!st || fails("copy")) return cudaErrorInvalidValue;
  to = d, from = s, count = n, pending = true;   // lands when the stream is waited for
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
  say("wait");
  if (pending) std::memcpy(to, from, count);
  pending = false;
  return cudaSuccess;
}
}
int main(int argc, char** argv) {
  if (argc > 1) fail_at = argv[1];
  const int table[4] = {3, 1, 4, 1};
  const int device = fails("device") ? 7 : 0;
  void* d = upload_table(device, table, sizeof(table));
  const bool there = d && !pending && std::memcmp(d, table, sizeof(table)) == 0;
  std::printf("table=%d dev=%d relaxed=%d\n", there, current, relaxed);
  int other[4] = {0, 0, 0, 0};
  const cudaError_t e = upload_bytes(device, other, table, sizeof(table));
  std::printf("bytes=%d dev=%d relaxed=%d\n", e == cudaSuccess && other[2] == 4, current, relaxed);
  if (d) std::free(d);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    if not os.path.exists(os.path.join(include, "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    d = tmp_path_factory.mktemp("upload")
    src, exe = d / "upload.cpp", d / "upload"
    src.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-x", "c++", str(src), "-o", str(exe), "-I", include, "-I",
                    os.path.join(ROOT, "bernsteinbasis.jl_gb300", "csrc")], check=True)
    return str(exe)


def lines(program, *args):
    out = subprocess.run([program, *args], check=True, capture_output=True, text=True).stdout
    return out.strip().splitlines()


def test_uploads_on_the_tables_device_and_waits(program):
    got = lines(program)
    assert got[:3] == ["malloc dev=0 relaxed=1", "copy dev=0 relaxed=1", "wait dev=0 relaxed=1"]
    # the caller's device and capture mode are back
    assert got[3] == "table=1 dev=1 relaxed=0" and got[-1] == "bytes=1 dev=1 relaxed=0"


@pytest.mark.parametrize("fault", ["malloc", "copy", "device"])
def test_failures_leave_nothing_behind(program, fault):
    got = lines(program, fault)
    assert "table=0 dev=1 relaxed=0" in got
    assert got[-1] == f"bytes={int(fault == 'malloc')} dev=1 relaxed=0"
    assert ("free dev=0 relaxed=1" in got) == (fault == "copy")
