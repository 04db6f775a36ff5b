// TMA copies of node-field boxes into shared memory, and the tensor maps that describe the fields.
#pragma once

#include <cuda.h>

#include "topx_kernels.cuh"

namespace topx {

// an array element at a byte offset (32 bits: no address arithmetic) from a uniform base
template <typename T, typename OFF>
__device__ __forceinline__ T* at(T* base, OFF bytes) {
  using C = typename std::conditional<std::is_const<T>::value, const char, char>::type;
  return reinterpret_cast<T*>(reinterpret_cast<C*>(base) + bytes);
}

__device__ __forceinline__ void tma_prefetch(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// One barrier per stage counts the bytes of its TMA copies.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return static_cast<unsigned>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint64_t* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
// waits for the phase of the given parity; false when it gave up, after about a second of the SM's clock
constexpr long long kWaitCycles = 1ll << 31;
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity) {
  if (mbar_try(b, parity)) return true;
  const long long t0 = clock64();
  do {
    if (mbar_try(b, parity)) return true;
  } while (clock64() - t0 < kWaitCycles);
  return false;
}
// A CTA's planes k = 0 .. last pass through two stages, each with its barrier, copied up to one plane ahead of the plane
// that is waited for.  False when the wait for plane k gave up: the thread that issues the copies has then waited
// once more for those in flight, and must issue no more, so that none lands after the CTA has ended.
__device__ __forceinline__ bool plane_wait(uint64_t* bar, int k, int last, bool issues) {
  if (mbar_wait(bar + (k & 1), unsigned(k) >> 1 & 1u)) return true;
  if (issues) {
    mbar_wait(bar + (k & 1), unsigned(k) >> 1 & 1u);
    if (k < last) mbar_wait(bar + (~k & 1), unsigned(k + 1) >> 1 & 1u);
  }
  return false;
}
// err: the engine's word for give-ups, in page-locked host memory (a host call that has synchronised reads it without a copy)
__device__ __forceinline__ void report_copy_wait(int* err) { *static_cast<volatile int*>(err) = kCoopErrCopy; }
// box of a 4-dimensional map (y, x, z, component) at (y, x, z, 0): entries outside the array read as zero.  y is
// even: a copy starts on a 16-byte boundary.
__device__ __forceinline__ void tma_load(void* dst, const CUtensorMap* map, int y, int x, int z, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(
          smem_addr(dst)),
      "l"(map), "r"(y), "r"(x), "r"(z), "r"(0), "r"(smem_addr(bar))
      : "memory");
}

// cuTensorMapEncodeTiled through the runtime (the library does not link the driver)
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    TOPX_CUDA_OK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q));
    if (!p || q != cudaDriverEntryPointSuccess) throw std::runtime_error("cuTensorMapEncodeTiled is not available");
    return reinterpret_cast<EncodeTiled>(p);
  }();
  return fn;
}

// map of ncomp node fields of the grid, boxes of by x bx nodes of one plane
template <typename T>
inline CUtensorMap field_map(const T* p, const Grid& g, int ncomp, int by, int bx) {
  constexpr bool f64 = sizeof(T) == 8;
  CUtensorMap m;
  const cuuint64_t dim[4] = {cuuint64_t(g.nny()), cuuint64_t(g.nnx()), cuuint64_t(g.nnz()), cuuint64_t(ncomp)};
  const cuuint64_t stride[3] = {sizeof(T) * dim[0], sizeof(T) * dim[0] * dim[1], sizeof(T) * cuuint64_t(g.stride)};
  const cuuint32_t box[4] = {cuuint32_t(by), cuuint32_t(bx), 1, cuuint32_t(ncomp)}, one[4] = {1, 1, 1, 1};
  if (encode_tiled()(&m, f64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<T*>(p), dim,
                     stride, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    throw std::runtime_error("cuTensorMapEncodeTiled failed");
  return m;
}

inline int num_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 148;
  return n > 0 ? n : 148;
}

}  // namespace topx
