// Order of the library's host calls on one context's buffers, without a GPU:
// db_api.cu and db_sgs.cu against a stand-in for the CUDA runtime that keeps,
// for every stream, the bytes its unfinished operations write.  Operations are
// unfinished until their stream is waited for; the legacy stream is not
// ordered with non-blocking streams, and a copy from pageable memory waits for
// the legacy stream before it starts but may land after the call returns.
// An operation on bytes that another stream still writes is a fault.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <vector>

#include "../diablo3_b200/csrc/db_kernels.cuh"
#include "../diablo3_b200/csrc/mlp.cuh"
#include "../include/diablo_b200.h"

namespace {
struct Span { const char* a; size_t n; };
std::map<cudaStream_t, std::vector<Span>> open_;   // unfinished writes (nullptr: the legacy stream)
std::map<char*, size_t> mem_;
int faults_ = 0;
std::string where_;

void touch(cudaStream_t st, const void* p, size_t n) {
  const char* a = (const char*)p;
  for (auto& s : open_)
    if (s.first != st)
      for (auto& w : s.second)
        if (a < w.a + w.n && w.a < a + n) {
          printf("%s: bytes that another stream still writes\n", where_.c_str());
          ++faults_;
          return;
        }
}
void write(cudaStream_t st, void* p, size_t n) {
  touch(st, p, n);
  open_[st].push_back({(const char*)p, n});
}
cudaStream_t stream_of(cudaStream_t s) { return s == cudaStreamLegacy ? nullptr : s; }
bool device(const void* p) {
  auto it = mem_.upper_bound((char*)p);
  return it != mem_.begin() && (--it, (char*)p < it->first + it->second);
}
// a kernel: it may read every buffer there is
cudaError_t kernel(cudaStream_t st) {
  for (auto& m : mem_) touch(st, m.first, m.second);
  return cudaSuccess;
}
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { mem_[(char*)(*p = malloc(n ? n : 1))] = n; return cudaSuccess; }
cudaError_t cudaFree(void* p) { open_.clear(); mem_.erase((char*)p); free(p); return cudaSuccess; }   // waits for the device
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int, size_t n) { write(nullptr, p, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int, size_t n, cudaStream_t s) { write(s, p, n); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  open_[nullptr].clear();
  if (k == cudaMemcpyHostToDevice) write(nullptr, d, n);
  else touch(nullptr, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  if (device(s)) touch(st, s, n);
  else if (device(d)) write(st, d, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { open_[stream_of(s)].clear(); return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { static uintptr_t k = 16; *s = (cudaStream_t)(k += 16); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return ""; }
}

// the kernels the calls below launch
namespace db {
struct SgsData;
cudaError_t launch_pfac(const Geom&, const State&, cudaStream_t st) { return kernel(st); }
cudaError_t launch_ref_to_spec(const Geom&, int, int, const double2*, double2*, cudaStream_t st) { return kernel(st); }
cudaError_t launch_inv_z(const Geom&, FieldSet, FieldSet, int, cudaStream_t st, unsigned, const double2*, double*) { return kernel(st); }
cudaError_t launch_inv_x(const Geom&, FieldSet, FieldSet, int, cudaStream_t st, unsigned) { return kernel(st); }
cudaError_t launch_sgs_targets(const Geom&, const State&, const SgsData&, cudaStream_t st) { return kernel(st); }
}  // namespace db
extern "C" cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms* p, cudaStream_t st) {
  if (device(p->dstPtr.ptr)) write(st, p->dstPtr.ptr, p->dstPtr.pitch * p->dstPtr.ysize * p->extent.depth);
  return cudaSuccess;
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  where_ = what;
  if (what == "sgs") {   // a network on a caller's non-blocking stream
    float v[DB_SGS_NPARAMS] = {}, one[16], lo[16], hi[16];
    for (int i = 0; i < 16; ++i) { one[i] = 1.f; lo[i] = -1.f; hi[i] = 1.f; }
    db_sgs_net* n = nullptr;
    if (db_sgs_create((void*)(uintptr_t)8, &n) || db_sgs_set_range(n, lo, hi) || db_sgs_set(n, v, lo, one, one) || db_sgs_get(n, v)) return 2;
    db_sgs_destroy(n);
  } else {               // a context on its own stream: creation and a first upload, training targets
    db_params p;
    memset(&p, 0, sizeof p);
    p.nx = p.nz = 16; p.ny = 9; p.n_th = 1; p.time_ad_meth = 1; p.re = p.pr = p.lx = p.lz = p.ro = p.delta = p.beta = 1.0;
    p.ly = 2.0; p.precision = what == "init mixed"; p.dthdx_override = NAN;
    double gy[10], gc[4 + 2];
    for (int i = 0; i < 10; ++i) gy[i] = -1.0 + 0.2 * i;
    for (int i = 0; i < 6; ++i) gc[i] = -1.0 + 0.4 * i;
    db_ctx* c = nullptr;
    if (db_init(&p, gy, nullptr, &c)) return 2;
    std::vector<double> f((size_t)2 * 9 * 18 * 11);
    if (db_upload_field(c, DB_CU1, f.data())) return 3;
    long long npts = 0;
    std::vector<float> out(1 << 16);
    if (what == "targets" && db_sgs_targets(c, 4, 2, 4, gc, out.data(), out.data(), &npts)) return 4;
    db_finalize(c);
  }
  printf("%s: %d faults\n", what.c_str(), faults_);
  return faults_ ? 1 : 0;
}
