"""The page-locked slots of large reads on the host alone: readback.cu compiled as C++ against a
runtime that counts, so that several devices can be told apart."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>
#include "b2b_internal.h"

static thread_local int current = 0;         // the device of the calling thread, as the runtime has it
static std::mutex m;
static std::map<void*, int> owner;           // allocations and the device they were made on
static int wrong = 0;
static cudaError_t make(void** p, size_t n) {
  *p = malloc(n);
  std::lock_guard<std::mutex> l(m);
  owner[*p] = current;
  return cudaSuccess;
}
static cudaError_t drop(void* p) {
  std::lock_guard<std::mutex> l(m);
  wrong += owner.at(p) != current;
  owner.erase(p);
  free(p);
  return cudaSuccess;
}
extern "C" {
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return make(p, n); }
cudaError_t cudaMalloc(void** p, size_t n) { return make(p, n); }
cudaError_t cudaFreeHost(void* p) { return drop(p); }
cudaError_t cudaFree(void* p) { return drop(p); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return make((void**)e, 1); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return cudaSuccess;
}
}

int main() {
  const size_t n = (5 << 20) + 12345;
  std::vector<unsigned char> value(n), read(n);
  for (size_t k = 0; k < n; ++k) value[k] = (unsigned char)(k * 2654435761u >> 13);
  b2b_net a{}, b{};
  a.cfg.device = 0;
  b.cfg.device = 1;
  b2b::readback_net_created();
  b2b::readback_net_created();
  // a few MB are one copy, without slots
  if (b2b::read_array(&a, read.data(), value.data(), 3 << 20) != cudaSuccess ||
      memcmp(read.data(), value.data(), 3 << 20) != 0 || !owner.empty())
    return 3;
  for (b2b_net* net : {&a, &b, &a}) {
    std::fill(read.begin(), read.end(), 0);
    cudaSetDevice(net->cfg.device);
    if (b2b::read_array(net, read.data(), value.data(), n) != cudaSuccess || read != value) return 1;
  }
  if (owner.empty()) return 2;               // a set of slots per device is kept for the next read
  cudaSetDevice(0);
  b2b::readback_net_destroyed();
  cudaSetDevice(3);
  b2b::readback_net_destroyed();             // the last net: the sets of devices 0 and 1 go
  printf("left %zu wrong %d device %d\n", owner.size(), wrong, current);
  return 0;
}
"""


def test_slots_of_every_device_go_and_the_callers_device_stays(tmp_path):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs the CUDA headers")
    src, exe = tmp_path / "slots.cpp", tmp_path / "slots"
    src.write_text(PROGRAM)
    csrc = os.path.join(ROOT, "brian2cuda_b200", "csrc")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CUDA}/include", f"-I{csrc}",
                    f"-I{ROOT}/include", str(src), "-x", "c++", os.path.join(csrc, "readback.cu"),
                    "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0
    assert out.stdout.split() == ["left", "0", "wrong", "0", "device", "3"]
