// Host code of the single-launch and batched solvers on a made-up device: what they launch, where, and what they do
// when a call fails. Linked with the solvers' objects and this file's CUDA runtime, which keeps a log and launches
// nothing. Arguments: the largest cluster that fits, the number of the call to fail (0: none) and its name, then
// "solve ROWS ENTRIES_A_ROW" or "batch ROWS...".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "femk_internal.cuh"

static int g_max_cluster = 16, g_fail_at = 0, g_calls = 0;
static const char* g_fail = "";
static cudaError_t call(const char* name) {
  if (g_fail_at && !strcmp(name, g_fail) && ++g_calls == g_fail_at) {
    printf("failed %s\n", name);
    return cudaErrorUnknown;
  }
  return cudaSuccess;
}
static int id(const void* handle) { return (int)(intptr_t)handle; }

#ifndef __CUDA_ARCH__  // the device pass has its own
extern "C" {
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made up"; }
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = calloc(1, n);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  memcpy(d, s, n);
  return call("cudaMemcpyAsync");
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  memset(d, v, n);
  return call("cudaMemsetAsync");
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return call("cudaFuncSetAttribute"); }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* cfg) {
  *n = cfg->attrs[0].val.clusterDim.x <= (unsigned)g_max_cluster ? 7 : 0;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  static intptr_t next = 100;
  *e = (cudaEvent_t)next++;
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  static intptr_t next = 10;
  *s = (cudaStream_t)next++;
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  const cudaError_t rc = call("cudaEventRecord");
  if (rc == cudaSuccess) printf("record %d %d\n", id(e), id(s));
  return rc;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
  const cudaError_t rc = call("cudaStreamWaitEvent");
  if (rc == cudaSuccess) printf("wait %d %d\n", id(s), id(e));
  return rc;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  printf("synchronize %d\n", id(s));
  return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* cfg, const void*, void**) {
  unsigned cluster = 0, coop = 0;
  for (unsigned i = 0; i < cfg->numAttrs; ++i) {
    if (cfg->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = cfg->attrs[i].val.clusterDim.x;
    if (cfg->attrs[i].id == cudaLaunchAttributeCooperative) coop = 1;
  }
  if (cluster > (unsigned)g_max_cluster) {
    printf("refused cluster %u\n", cluster);
    return cudaErrorUnknown;
  }
  const cudaError_t rc = call("cudaLaunchKernelExC");
  if (rc == cudaSuccess) printf("launch %d blocks %u cluster %u cooperative %u\n", id(cfg->stream), cfg->gridDim.x, cluster, coop);
  return rc;
}
}
#endif

namespace femk {
void set_error(const std::string& m) { printf("error %s\n", m.c_str()); }
void clear_error() {}
int counted_launch() { return 0; }
int ensure_workspace(femk_plan* p) {
  if (!p->work) p->work = (double*)calloc(5 * p->vstride, 8);
  return FEMK_OK;
}
int ensure_sell_values(femk_plan*, bool) { return FEMK_OK; }
int launch_sell_values(const femk_plan*, const double*, bool, cudaStream_t) { return FEMK_OK; }
int check_bounds(const femk_plan*, cudaStream_t, const char*) {
  printf("checked\n");
  return FEMK_OK;
}
}  // namespace femk

int main(int argc, char** argv) {
  using namespace femk;
  g_max_cluster = atoi(argv[1]);
  g_fail_at = atoi(argv[2]);
  g_fail = argv[3];
  const cudaStream_t s = (cudaStream_t)(intptr_t)1;
  femk_plan p;
  std::vector<int64_t> off{0};
  const bool batch = !strcmp(argv[4], "batch");
  for (int i = 5; i < (batch ? argc : 6); ++i) off.push_back(off.back() + atoll(argv[i]));
  const int64_t entries = batch ? 15 : atoll(argv[6]);
  p.n = off.back();
  p.n_slices = (p.n + 31) / 32;
  p.sell_nnz = 32 * entries * p.n_slices;
  p.vstride = (p.n + 63) & ~int64_t(63);
  p.n_sm = 148;
  p.coop = p.persist_ok = 1;
  p.order = 1;
  p.barrier_spin = 1000;
  p.sell_cols = (int32_t*)1;
  p.sell_c16 = (int16_t*)1;
  std::vector<double> v(p.n);
  int rc = 0;
  if (batch) {
    printf("sets %d\n", (int)batch_sets_fit(&p, (int32_t)off.size() - 1, off.data()));
    rc = batch_sets(&p, (int32_t)off.size() - 1, off.data(), v.data(), v.data(), v.data(), nullptr, 1e-8, 0.0, 10,
                    nullptr, nullptr, nullptr, s);
  } else {
    int32_t it = 0;
    double rel = 0.0;
    rc = pcg_persist(&p, v.data(), v.data(), v.data(), nullptr, 1e-8, 0.0, 10, &it, &rel, s);
    printf("status %d\n", rc);
    BicgResult out{};
    std::vector<double> ws(8 * p.vstride);
    rc = bicg_persist(&p, v.data(), v.data(), nullptr, ws.data(), 1e-8, 0.0, 10, s, &out);
  }
  printf("status %d\n", rc);
  return 0;
}
