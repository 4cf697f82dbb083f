"""The buffer pool (csrc/pool.cu) against a model of the driver's allocator: a device
of a few megabytes, streams that can be capturing, frees that can fail. Compiled for the
CPU, so that running out of memory and contexts in the middle of a capture cost nothing."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CUDA = next((p for p in (Path("/usr/local/cuda/include"),) if (p / "cuda_runtime.h").exists()), None)

MODEL = r'''
#include "pool.cu"
#include <cstdio>
#include <set>
namespace {
constexpr size_t MB = 1 << 20;
struct Device { size_t capacity = 0, reserved = 0, used = 0; } dev[2];
struct Stream { int device; bool capturing = false; int frees = 0; } st[4];
std::map<void*, std::pair<int, size_t>> live;
int fail_frees = 0, bad = 0;
Stream& of(cudaStream_t s) { return st[(size_t)s - 1]; }
cudaStream_t stream(int i) { return (cudaStream_t)(size_t)(i + 1); }
void expect(bool ok, const char* what) {
  if (!ok) { std::printf("failed: %s\n", what); ++bad; }
}
}
extern "C" {
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t s) {
  Device& d = dev[of(s).device];
  if (d.used + n > d.capacity) return cudaErrorMemoryAllocation;
  d.used += n;
  if (d.used > d.reserved) d.reserved = d.used;
  static size_t next = 4096;
  *p = (void*)next; next += n + 4096;
  live[*p] = {of(s).device, n};
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  if (fail_frees > 0) { --fail_frees; return cudaErrorUnknown; }
  ++of(s).frees;
  if (of(s).capturing) return cudaErrorStreamCaptureInvalidated;
  if (!live.count(p)) { std::printf("failed: freed twice\n"); ++bad; return cudaErrorInvalidValue; }
  dev[live[p].first].used -= live[p].second;
  live.erase(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  expect(!of(s).capturing, "a capturing stream is not synchronised");
  return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
  *c = of(s).capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
  *t = dev[0].capacity; *f = dev[0].capacity - dev[0].reserved; return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int d) {
  *p = (cudaMemPool_t)(size_t)(d + 1); return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  const Device& d = dev[(size_t)p - 1];
  *(uint64_t*)v = a == cudaMemPoolAttrReservedMemCurrent ? d.reserved : d.used;
  return cudaSuccess;
}
}
namespace evoc {
[[noreturn]] void throw_cuda(cudaError_t, const char* what, const char*, int) { throw Error(1, what); }
}
using namespace evoc;
namespace {
DevBuf<char> take(int s, size_t mb) { return DevBuf<char>(mb * MB, stream(s)); }
// A pool of ctx `s` that holds mb free megabytes in blocks of one.
void fill(int s, int mb) {
  std::vector<DevBuf<char>> b;
  for (int i = 0; i < mb; ++i) b.push_back(take(s, 1));
}
void open(int s, int device, size_t limit) { st[s].device = device; dev_pool_open(stream(s), device, limit); }
SCENARIO
}
int main() { scenario(); std::printf(bad ? "bad\n" : "ok\n"); return bad; }
'''

SCENARIOS = {
    # another context's pool is given back for an allocation, but never into its capture
    "capture": r'''
void scenario() {
  dev[0].capacity = 64 * MB;
  open(0, 0, 40 * MB); open(1, 0, 40 * MB);
  fill(1, 32);
  for (int by_library = 0; by_library < 2; ++by_library) {
    st[1].capturing = true;
    if (by_library) dev_pool_capture(stream(1), true);
    bool refused = false;
    try { take(0, 48); } catch (const Error&) { refused = true; }
    expect(refused, "nothing to be had while the other context captures");
    expect(st[1].frees == 0, "no free on a capturing stream");
    expect(dev_pool_bytes(stream(1)) == 32 * MB, "its pool is whole");
    st[1].capturing = false;
    if (by_library) dev_pool_capture(stream(1), false);
  }
  // flagged before the stream itself says so: the capture is about to begin
  dev_pool_capture(stream(1), true);
  try { take(0, 48); } catch (const Error&) {}
  expect(st[1].frees == 0, "no free once a capture is announced");
  dev_pool_capture(stream(1), false);
  DevBuf<char> b = take(0, 48);
  expect(b.get() != nullptr && st[1].frees == 32, "given up afterwards");
}''',
    # what can be had is the same before a buffer's first use and after its free, whether
    # the free put it into this pool, another one or the driver's
    "available": r'''
void scenario() {
  dev[0].capacity = 64 * MB;
  open(0, 0, 8 * MB); open(1, 0, 8 * MB);
  expect(dev_available(stream(0)) == 64 * MB, "all of it");
  for (int round = 0; round < 3; ++round) {  // a plan built, freed and built again
    expect(30 * MB <= dev_available(stream(0)) / 2, "half of it is enough for the slots");
    { DevBuf<char> slots = take(0, 30); expect(dev_available(stream(0)) == 34 * MB, "in use"); }
    expect(dev_available(stream(0)) == 64 * MB, "above the bound: back with the driver's pool");
  }
  fill(0, 8); fill(0, 4); fill(1, 8);
  { DevBuf<char> b = take(0, 6); }  // evicts
  expect(dev_available(stream(0)) == 64 * MB, "in this pool and the other's");
  DevBuf<char> b = take(1, 20);
  expect(dev_available(stream(0)) == 44 * MB, "less what is in use");
}''',
    "devices": r'''
void scenario() {
  dev[0].capacity = dev[1].capacity = 16 * MB;
  open(0, 0, 16 * MB); open(1, 1, 16 * MB);
  fill(1, 8);
  bool refused = false;
  try { take(0, 20); } catch (const Error&) { refused = true; }
  expect(refused && st[1].frees == 0, "a pool on another device is of no use");
  expect(dev_available(stream(0)) == 16 * MB, "nor is it counted");
}''',
    # a buffer that cannot be freed is kept, not lost
    "failing_free": r'''
void scenario() {
  dev[0].capacity = 64 * MB;
  open(0, 0, 8 * MB);
  fill(0, 8);
  fail_frees = 1;
  { DevBuf<char> b = take(0, 2); }  // over the bound: the oldest has to go, and cannot
  expect(dev_pool_bytes(stream(0)) == 10 * MB && live.size() == 9, "kept when its free fails");
  { DevBuf<char> b = take(0, 3); }
  expect(dev_pool_bytes(stream(0)) <= 8 * MB, "back under the bound with the next");
  dev_pool_close(stream(0));
  expect(live.empty(), "all given back with the context");
}''',
    # a buffer above the bound goes to the driver; evictions take the oldest
    "bound": r'''
void scenario() {
  dev[0].capacity = 64 * MB;
  open(0, 0, 8 * MB);
  { DevBuf<char> b = take(0, 12); }
  expect(dev_pool_bytes(stream(0)) == 0 && live.empty(), "above the bound: not kept");
  fill(0, 8);
  { DevBuf<char> b = take(0, 4); }
  expect(dev_pool_bytes(stream(0)) == 8 * MB && live.size() == 5, "four of one made room for four");
}''',
}


@pytest.mark.parametrize("name", sorted(SCENARIOS))
def test_pool(name, tmp_path):
    if CUDA is None or not shutil.which("g++"):
        pytest.skip("CUDA headers or g++ missing")
    src = tmp_path / "model.cpp"
    src.write_text(MODEL.replace("SCENARIO", SCENARIOS[name]))
    exe = tmp_path / "model"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CUDA}", f"-I{ROOT / 'evoc-rs_gb300' / 'csrc'}",
                    str(src), "-o", str(exe)], check=True, capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout
