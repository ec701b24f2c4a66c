// Row-wise joins and activations in two forms: for few rows, which are bound by one block's chain of trips, and for many,
// which are bound by bytes in flight.
#pragma once

#include "common.cuh"

// A launch of up to FEW_ROWS rows is (where the caller's `pdl` asks for it) a programmatic dependent: its blocks come in, and fetch the
// layer's own numbers, while the launch before it drains; the kernel waits before it reads or writes what other launches touch, and
// reads that past L1 (ld_prev).  The rows are those up to which the products on both sides overlap their launches too.  Up to FORM_ROWS
// rows take the same form as ordinary launches (four streams of 2,048 columns: 64 rows 4.3 us against 4.9; 300 rows 10 against 6).
constexpr int FEW_ROWS = 16, FORM_ROWS = 64;

template <typename... P, typename... A>
static int launch_rows(void (*kern)(P...), dim3 grid, int threads, size_t smem, bool behind, cudaStream_t st, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = behind ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, (P)a...);
  return e != cudaSuccess ? (int)e : launch_status();
}
__device__ __forceinline__ void wait_for_earlier_launches() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// An earlier launch's results: one element, or four consecutive ones at once (8 or 16 bytes).  FEW: past L1.
template <bool FEW, typename V> __device__ __forceinline__ V load_word(const V* p) { return FEW ? ld_prev(p) : *p; }
template <bool FEW> __device__ __forceinline__ float4 load4(const float* p) { return load_word<FEW>(reinterpret_cast<const float4*>(p)); }
template <bool FEW> __device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 raw = load_word<FEW>(reinterpret_cast<const uint2*>(p));
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), b = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
template <bool FEW> __device__ __forceinline__ float load1(const float* p) { return load_word<FEW>(p); }
template <bool FEW> __device__ __forceinline__ float load1(const __nv_bfloat16* p) { return FEW ? ld_prev_bf16(p) : to_f32(*p); }
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 raw;
  raw.x = *reinterpret_cast<unsigned*>(&a);
  raw.y = *reinterpret_cast<unsigned*>(&b);
  *reinterpret_cast<uint2*>(p) = raw;
}

// A block's row is summed in the order of ROW_THREADS threads in both forms, so that its result does not depend on how many rows there
// are.  The form for few rows brings a row wider than 1,024 in with twice the threads (2,048 columns: one trip to memory instead of two)
// and sums what they left in shared memory with the first half; for many rows blocks of 512 would leave an SM with one or two of
// them (four streams of 2,048 columns, 2,048 rows, bfloat16: 48 us against 27).
constexpr int ROW_THREADS = 256, WIDE_ROW = 1024;
