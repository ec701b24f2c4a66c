// Mixture of experts for many tokens (bfloat16): the assignments (token, k) sorted by expert, and the experts' two
// products as grouped tensor-core products over the sorted rows.  Everything is decided on the device: no count ever
// reaches the host, so a step with these launches can be captured in a graph.
//
//   moe_sort       counts per expert -> the sorted place of every assignment (the order inside an expert
//                  is arbitrary: every row is computed on its own, so no result depends on it); the list of row tiles
//                  (expert, first sorted place, rows) that the products walk, and their number.  One block.
//   moe_gather     xs[place] = its token's row, perm[place] = the assignment
//   first product  act[p, f] = silu(Wg_e[f] . h[token(p)]) * (Wu_e[f] . h[token(p)])
//   second product y[perm[p], c] = Wd_e[c] . act[p]                                   rows scattered back
//
// Inner sizes that are multiples of 64 run on tcgen05 (moe_grouped_tc_kernel), with the sorted rows gathered first
// (moe_gather); other multiples of 16 run on mma.sync (moe_grouped_kernel): a block of four warps computes 64 or 128 sorted
// rows of one expert x 128 weight rows, operands through a two-stage cp.async ring of 64-wide k slices, rows gathered through
// the permutation on their way in, what does not exist filled with zeros.
//
// No block waits on another block.
#include "common.cuh"
#include "drain.h"
#include <cuda.h>
#include <atomic>
#include <math.h>
#include <type_traits>

namespace {
typedef __nv_bfloat16 bf16;
constexpr int BK = 64;                    // k slice
constexpr int LDS = BK + 8;               // padded row stride (elements): conflict-free ldmatrix
constexpr int STAGES = 2;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int bytes) {
  unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }
__device__ __forceinline__ void ldsm_x4(unsigned& r0, unsigned& r1, unsigned& r2, unsigned& r3, const void* p) {
  unsigned s = (unsigned)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(s));
}
__device__ __forceinline__ void mma16816(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}

constexpr int SORT_THREADS = 1024, SORT_INTS = 12 * 1024 /* 48 KB of counters */, SORT_KEEP = 16;

// Warps count into `hists` tables of their own (32 while E <= 372), so that atomics on a popular expert's counter collide
// inside a warp only, and scatter through the same tables: 16,384 assignments to 64 experts take 7.7 us where one table took 19.
// What leaves is `place[assignment]` or, where that is null, `perm[place]`.  Rows of an expert are cut into equal tiles of up to `BM`,
// rounded up to 16; tiles of more than BM / 2 rows come first in the list (blocks that draw their work draw the long pieces first).
// `next`: the products' counters of work drawn, set to zero.
__global__ void __launch_bounds__(SORT_THREADS) moe_sort_kernel(
    const int* __restrict__ idx, int n_assign, int E, int BM, int hists, int* __restrict__ perm, int* __restrict__ place,
    int* __restrict__ tile_expert, int* __restrict__ tile_row0, int* __restrict__ tile_rows, int* __restrict__ n_tiles,
    int* __restrict__ next) {
  extern __shared__ int sh[];   // [hists][E] counters, then cursors; [E] offsets
  int* const mine = sh + (size_t)((threadIdx.x >> 5) % hists) * E;
  int* const first = sh + (size_t)hists * E;
  for (int i = threadIdx.x; i < hists * E; i += SORT_THREADS) sh[i] = 0;
  __syncthreads();
  // a thread's assignments are requested together, and kept for the scatter where they are no more than SORT_KEEP
  int kept[SORT_KEEP];
  for (int a0 = threadIdx.x; a0 < n_assign; a0 += SORT_KEEP * SORT_THREADS) {
#pragma unroll
    for (int i = 0; i < SORT_KEEP; ++i) kept[i] = a0 + i * SORT_THREADS < n_assign ? min(max(idx[a0 + i * SORT_THREADS], 0), E - 1) : -1;
#pragma unroll
    for (int i = 0; i < SORT_KEEP; ++i)
      if (kept[i] >= 0) atomicAdd(&mine[kept[i]], 1);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += SORT_THREADS) {
    int run = 0;
    for (int w = 0; w < hists; ++w) run += sh[(size_t)w * E + e];
    first[e] = run;
  }
  __syncthreads();
  if (threadIdx.x < 32) {       // offsets and tiles: a scan over the experts by one warp
    const int lane = threadIdx.x;
    auto tiles_of = [&](int c) { return (c + BM - 1) / BM; };
    auto per_of = [&](int c, int t) { return t ? ((c + t - 1) / t + 15) / 16 * 16 : 0; };      // `t` tiles of so many rows, none empty
    auto large = [&](int per) { return 2 * per > BM; };
    int n_large = 0;
    for (int e = lane; e < E; e += 32) {
      const int t = tiles_of(first[e]);
      if (large(per_of(first[e], t))) n_large += t;
    }
    for (int o = 16; o > 0; o >>= 1) n_large += __shfl_xor_sync(0xffffffffu, n_large, o);
    int rows_before = 0, large_before = 0, small_before = n_large;      // the list starts with the large tiles
    for (int e0 = 0; e0 < E; e0 += 32) {
      const int e = e0 + lane, c = e < E ? first[e] : 0, t = tiles_of(c), per = per_of(c, t);
      const bool big = large(per);
      int rs = c, ls = big ? t : 0, ss = big ? 0 : t;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int r2 = __shfl_up_sync(0xffffffffu, rs, o), l2 = __shfl_up_sync(0xffffffffu, ls, o), s2 = __shfl_up_sync(0xffffffffu, ss, o);
        if (lane >= o) { rs += r2; ls += l2; ss += s2; }
      }
      const int row0 = rows_before + rs - c, tile0 = big ? large_before + ls - t : small_before + ss - t;
      if (e < E) {
        first[e] = row0;
        for (int i = 0; i < t; ++i) {
          tile_expert[tile0 + i] = e;
          tile_row0[tile0 + i] = row0 + i * per;
          tile_rows[tile0 + i] = min(per, c - i * per);
        }
      }
      rows_before += __shfl_sync(0xffffffffu, rs, 31);
      large_before += __shfl_sync(0xffffffffu, ls, 31);
      small_before += __shfl_sync(0xffffffffu, ss, 31);
    }
    if (lane == 0) { *n_tiles = small_before; next[0] = next[1] = 0; }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += SORT_THREADS) {
    int run = first[e];
    for (int w = 0; w < hists; ++w) {
      const int c = sh[(size_t)w * E + e];
      sh[(size_t)w * E + e] = run;
      run += c;
    }
  }
  __syncthreads();
  for (int a0 = threadIdx.x; a0 < n_assign; a0 += SORT_KEEP * SORT_THREADS) {
    if (n_assign > SORT_KEEP * SORT_THREADS) {
#pragma unroll
      for (int i = 0; i < SORT_KEEP; ++i) kept[i] = a0 + i * SORT_THREADS < n_assign ? min(max(idx[a0 + i * SORT_THREADS], 0), E - 1) : -1;
    }
#pragma unroll
    for (int i = 0; i < SORT_KEEP; ++i)
      if (kept[i] >= 0) {
        const int at = atomicAdd(&mine[kept[i]], 1);
        if (place) place[a0 + i * SORT_THREADS] = at;      // in order: one SM's scattered stores of `perm` cost as much as the rest
        else perm[at] = a0 + i * SORT_THREADS;
      }
  }
}

// MODE 0: A rows are h[perm[p] / top], B is W_gu[e] ([2F, K]: gate rows then up rows), out is act[p, F]
// MODE 1: A rows are act[p],           B is W_d[e]  ([C, K]),                        out is y[perm[p], C]
// MODE 2: A rows are h[perm[p] / top], B is W_u[e]  ([F, K]: experts without a gate), out is act[p, F] = max(., 0)^2
// MODE 3: as MODE 0 with the assignment's weight on the expert's INPUT and a clamped activation: with s = in_w[perm[p]],
//         g = min(s * gate, limit), u = clamp(s * up, -limit, limit), act[p, f] = g * sigmoid(alpha * g) * (u + up_off)
// A block of 2 x 2 warps computes BM sorted rows x BN output columns (of gate AND up in mode 0), a warp BM/2 x BN/2.
template <int MODE, int BM, int BN>
__global__ void __launch_bounds__(128) moe_grouped_kernel(
    const bf16* __restrict__ a_in, const bf16* __restrict__ w, const int* __restrict__ perm,
    const int* __restrict__ tile_expert, const int* __restrict__ tile_row0, const int* __restrict__ tile_rows,
    const int* __restrict__ n_tiles, int top, int K, int n_out, bf16* __restrict__ out, const float* __restrict__ in_w, float limit, float alpha, float up_off) {
  constexpr int NTHREADS = 128;
  constexpr int NMAT = (MODE == 0 || MODE == 3) ? 2 : 1;       // weight matrices multiplied at once (gate and up)
  constexpr int NB = NMAT * BN;                 // weight rows a block reads per k slice
  constexpr int WM = BM / 2, WN = BN / 2;       // a warp's rows and columns
  constexpr int MT = WM / 16, NT = WN / 8;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* as = reinterpret_cast<bf16*>(smem_raw);   // [STAGES][BM][LDS]
  bf16* bs = as + STAGES * BM * LDS;              // [STAGES][NB][LDS]
  __shared__ int row_src[BM];

  const int tile = blockIdx.x;
  if (tile >= *n_tiles) return;
  const int e = tile_expert[tile], p0 = tile_row0[tile];
  const int rows = tile_rows[tile];
  const int n0 = blockIdx.y * BN;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int wm = warp >> 1, wn = warp & 1;
  const int g = lane >> 2, t = lane & 3;

  for (int r = tid; r < BM; r += NTHREADS) row_src[r] = r < rows ? (MODE != 1 ? perm[p0 + r] / top : p0 + r) : -1;
  __syncthreads();
  const bf16* we = w + (size_t)e * (NMAT * n_out) * K;

  auto load = [&](int stage, int k0) {
    bf16* a_st = as + stage * BM * LDS;
    bf16* b_st = bs + stage * NB * LDS;
    constexpr int CPR = BK / 8;
    for (int i = tid; i < BM * CPR; i += NTHREADS) {
      const int r = i / CPR, c = i % CPR;
      const int src = row_src[r];
      const bool ok = src >= 0 && k0 + c * 8 < K;
      cp_async16(a_st + r * LDS + c * 8, a_in + (ok ? (size_t)src * K + k0 + c * 8 : 0), ok ? 16 : 0);
    }
    for (int i = tid; i < NB * CPR; i += NTHREADS) {
      const int r = i / CPR, c = i % CPR;
      int wr = n0 + (r % BN);
      const bool ok = wr < n_out && k0 + c * 8 < K;
      if ((MODE == 0 || MODE == 3) && r >= BN) wr += n_out;   // the matching up rows
      cp_async16(b_st + r * LDS + c * 8, we + (ok ? (size_t)wr * K + k0 + c * 8 : 0), ok ? 16 : 0);
    }
  };

  float acc[NMAT][MT][NT][4];
#pragma unroll
  for (int m = 0; m < NMAT; ++m)
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[m][i][j][x] = 0.f;

  // a ring of STAGES k slices: slice s + STAGES - 1 is requested while slice s is multiplied; one group is committed per
  // step whether or not it holds a slice, so that the number of groups in flight names the slice that has landed
  const int nk = (K + BK - 1) / BK;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < nk) load(s, s * BK);
    cp_async_commit();
  }
  for (int ks = 0; ks < nk; ++ks) {
    cp_async_wait<STAGES - 2>();
    __syncthreads();   // slice ks has landed for every thread, and every warp is done with the stage refilled next
    if (ks + STAGES - 1 < nk) load((ks + STAGES - 1) % STAGES, (ks + STAGES - 1) * BK);
    cp_async_commit();
    const bf16* a_st = as + (ks % STAGES) * BM * LDS;
    const bf16* b_st = bs + (ks % STAGES) * NB * LDS;
#pragma unroll
    for (int kk = 0; kk < BK / 16; ++kk) {
      unsigned a[MT][4];
#pragma unroll
      for (int i = 0; i < MT; ++i)
        ldsm_x4(a[i][0], a[i][1], a[i][2], a[i][3], a_st + (wm * WM + i * 16 + (lane & 15)) * LDS + kk * 16 + (lane >> 4) * 8);
#pragma unroll
      for (int m = 0; m < NMAT; ++m) {
#pragma unroll
        for (int j = 0; j < NT; j += 2) {
          unsigned b0, b1, b2, b3;
          ldsm_x4(b0, b1, b2, b3, b_st + (m * BN + wn * WN + j * 8 + (lane & 7) + (lane >> 4) * 8) * LDS + kk * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            mma16816(acc[m][i][j], a[i][0], a[i][1], a[i][2], a[i][3], b0, b1);
            mma16816(acc[m][i][j + 1], a[i][0], a[i][1], a[i][2], a[i][3], b2, b3);
          }
        }
      }
    }
  }
  cp_async_wait<0>();

#pragma unroll
  for (int i = 0; i < MT; ++i) {
    const int r0 = wm * WM + i * 16 + g, r1 = r0 + 8;
    size_t o0 = 0, o1 = 0;
    if (MODE != 1) {
      o0 = (size_t)(p0 + r0) * n_out;
      o1 = (size_t)(p0 + r1) * n_out;
    } else {
      if (r0 < rows) o0 = (size_t)perm[p0 + r0] * n_out;
      if (r1 < rows) o1 = (size_t)perm[p0 + r1] * n_out;
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const int c = n0 + wn * WN + j * 8 + 2 * t;
      if (c >= n_out) continue;     // n_out is even (a multiple of 16): c + 1 is inside too
      float v0 = acc[0][i][j][0], v1 = acc[0][i][j][1], v2 = acc[0][i][j][2], v3 = acc[0][i][j][3];
      if (MODE == 0) {
        v0 = v0 / (1.f + expf(-v0)) * acc[NMAT - 1][i][j][0];
        v1 = v1 / (1.f + expf(-v1)) * acc[NMAT - 1][i][j][1];
        v2 = v2 / (1.f + expf(-v2)) * acc[NMAT - 1][i][j][2];
        v3 = v3 / (1.f + expf(-v3)) * acc[NMAT - 1][i][j][3];
      }
      if (MODE == 3) {
        const float s0 = r0 < rows ? in_w[perm[p0 + r0]] : 0.f, s1 = r1 < rows ? in_w[perm[p0 + r1]] : 0.f;
        const float sc[4] = {s0, s0, s1, s1};
        float* v[4] = {&v0, &v1, &v2, &v3};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float gq = fminf(*v[q] * sc[q], limit);
          const float uq = fminf(fmaxf(acc[NMAT - 1][i][j][q] * sc[q], -limit), limit);
          *v[q] = gq / (1.f + expf(-alpha * gq)) * (uq + up_off);
        }
      }
      if (MODE == 2) {
        v0 = fmaxf(v0, 0.f); v1 = fmaxf(v1, 0.f); v2 = fmaxf(v2, 0.f); v3 = fmaxf(v3, 0.f);
        v0 *= v0; v1 *= v1; v2 *= v2; v3 *= v3;
      }
      if (r0 < rows) *reinterpret_cast<unsigned*>(out + o0 + c) = pack_bf16(v0, v1);
      if (r1 < rows) *reinterpret_cast<unsigned*>(out + o1 + c) = pack_bf16(v2, v3);
    }
  }
}

template <int MODE, int BM, int BN>
int gemm_launch(const void* a_in, const void* w, const int* perm, const int* tile_expert, const int* tile_row0, const int* tile_rows,
                const int* n_tiles, int top, int K, int n_out, void* out, int max_tiles, cudaStream_t st,
                const float* in_w = nullptr, float limit = 0.f, float alpha = 1.f, float up_off = 0.f) {
  static bool attr_set = false;   // set by the first (eager) launch, outside any stream capture
  constexpr size_t smem = sizeof(bf16) * (size_t)LDS * STAGES * (BM + ((MODE == 0 || MODE == 3) ? 2 * BN : BN));
  if (smem > 48 * 1024 && !attr_set) {
    cudaError_t e = cudaFuncSetAttribute(moe_grouped_kernel<MODE, BM, BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const int n_tiles_n = (n_out + BN - 1) / BN;
  if (n_tiles_n > 65535) return DRYFT_ERR_UNSUPPORTED;
  dim3 grid(max_tiles, n_tiles_n);
  moe_grouped_kernel<MODE, BM, BN><<<grid, 128, smem, st>>>((const bf16*)a_in, (const bf16*)w, perm, tile_expert, tile_row0, tile_rows,
                                                          n_tiles, top, K, n_out, (bf16*)out, in_w, limit, alpha, up_off);
  return launch_status();
}

// ---------------------------------------------------------------------------- tcgen05
// xs[place[a]] = h[a / top]: the sorted rows as one matrix that the copy engine takes in boxes (a copy of its own for each row's
// 128 bytes is bound by the engine's request rate).  A warp a row; it leaves perm[place[a]] = a beside it.
template <bool SIGNAL>
__global__ void __launch_bounds__(256) moe_gather_kernel(const uint4* __restrict__ h, const int* __restrict__ place, int n_assign, int top,
                                                         int per_row, uint4* __restrict__ xs, int* __restrict__ perm) {
  if (SIGNAL) let_next_launch_in();
  const int a = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (a >= n_assign) return;
  const int p = place[a];
  if (lane == 0) perm[p] = a;
  const uint4* from = h + (size_t)(a / top) * per_row;
  uint4* to = xs + (size_t)p * per_row;
#pragma unroll 8
  for (int c = lane; c < per_row; c += 32) to[c] = from[c];
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(void* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(void* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(void* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(void* bar, unsigned parity) {
  unsigned ok;
  asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
constexpr long long WAIT_CYCLES = 2000000000LL;   // about a second: then the waiter raises *err and every role gives up
__device__ __forceinline__ bool mbar_wait(void* bar, unsigned parity, int* err, volatile int* failed, int place) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (*failed) return false;
    if (clock64() - t0 > WAIT_CYCLES) {
      if (err) atomicCAS(err, 0, 200 + place);
      *failed = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, void* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y) : "memory");
}
// K-major operand tile, 128-byte swizzle: rows of 64 bf16 (128 bytes), 8-row groups 1024 bytes apart
__device__ __forceinline__ unsigned long long umma_desc(const void* smem_tile) {
  return (unsigned long long)((smem_u32(smem_tile) & 0x3FFFF) >> 4) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma(unsigned d_tmem, unsigned long long a_desc, unsigned long long b_desc, unsigned id, unsigned accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(id), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(void* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}

// n / (1 + e) for e >= 0: the quotient by an approximate reciprocal, and one of Newton's corrections of it by what is left of n; quarters of
// both, so that the reciprocal of a sum beyond 2^126 is still a normal number.  Without a branch, so that a thread's sixteen quotients
// overlap: with the compiler's division, which branches for extreme exponents, a layer of 64 experts of 768 x 2,048 takes 280 us for
// 2,048 tokens x 8, with this one 262.  For silu of every gate between -88.7 and 200 the two give the same 32-bit values, 4.2 x 2^-24 off at
// most; a fast exponential and division (258 us) are 18 x 2^-24 off and give zero below -87.3.
__device__ __forceinline__ float over_one_plus(float n, float e) {
  const float d = fmaf(e, 0.25f, 0.25f), m = 0.25f * n;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  const float q = m * r, better = fmaf(fmaf(-q, d, m), r, q);
  return better == better ? better : q;      // infinite n or e: nothing to correct
}

// The product is computed transposed: two tiles of 128 weight rows (gate and up rows of the same 128 features, or 256
// features) are the 128-row operands, up to NMAX sorted rows of one expert the columns, so that an expert's last tile is
// padded to 16 rows and not to 128.  What bounds it: operands on their way from L2 (a k slice of 64 is 32 KB of weights and
// up to 32 KB of rows for 8.4 Mflop; a copy of the rows is read by every feature tile).  One persistent block an SM draws
// (row tile, feature tile) units from a counter, the copies of the next unit on their way while one is finished; a unit's
// number goes from warp to warp behind the barriers that its data goes through (-1: no more).
//   warp 0 (one thread)  copies: weights 128 x 64 twice, rows in boxes of 64 x 64
//   warp 1 (one thread)  tcgen05.mma, accumulators 512 columns of tensor memory: with NMAX = 128 two units' worth
//   warps 2-9            read a unit's sums (lane = feature, column = sorted row), activation, store; neighbouring lanes swap
//                        so that a lane stores two features of one row
// MODE as in moe_grouped_kernel.  2,048 tokens x 8 of 64 experts of 768 x 2,048, each alone and cold: 132 us for the first product (0.78
// PFLOP/s), 86 for the second, where mma.sync takes 447 and 207.
template <int MODE, int NMAX> struct Tc {
  static constexpr bool GATED = MODE == 0 || MODE == 3;
  static constexpr int FEATURES = GATED ? 128 : 256;          // output features of a unit
  static constexpr int W_BYTES = 2 * 128 * 64 * 2, X_BYTES = NMAX * 64 * 2;
  static constexpr int STAGE_BYTES = W_BYTES + X_BYTES;
  static constexpr int STAGES = NMAX == 256 ? 3 : 4;
  static constexpr int BUFS = 256 / NMAX;
  static constexpr int BARS = 2 * STAGES + 2 * BUFS;
  static constexpr int RING = 16;       // unit numbers: more than units can be on their way (STAGES + BUFS + 1)
  static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + 8 * BARS + 16 + 4 * RING;
};
constexpr int TC_THREADS = 320;

template <int MODE, int NMAX>
__global__ void __launch_bounds__(TC_THREADS) moe_grouped_tc_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const int* __restrict__ perm,
    const int* __restrict__ tile_expert, const int* __restrict__ tile_row0, const int* __restrict__ tile_rows,
    const int* __restrict__ n_tiles, int* __restrict__ next, int n_kb, int n_out, int f_tiles, bf16* __restrict__ out,
    const float* __restrict__ in_w, float limit, float alpha, float up_off, int* err) {
  typedef Tc<MODE, NMAX> L;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* const stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned long long* const full = reinterpret_cast<unsigned long long*>(stages + L::STAGES * L::STAGE_BYTES);
  unsigned long long* const empty = full + L::STAGES;
  unsigned long long* const acc_full = empty + L::STAGES;
  unsigned long long* const acc_empty = acc_full + L::BUFS;
  unsigned* const tmem_slot = reinterpret_cast<unsigned*>(acc_empty + L::BUFS);
  volatile int* const ring = reinterpret_cast<volatile int*>(tmem_slot + 4);
  __shared__ int failed_s, issued_s;                  // issued_s: stages that the copying thread has filled or closed
  __shared__ unsigned long long drained_s;            // after a failure: the products issued so far are done
  volatile int* failed = &failed_s;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows_per_expert = L::GATED ? 2 * n_out : n_out;

  if (threadIdx.x == 0) {
    failed_s = issued_s = 0;
    mbar_init(&drained_s, 1);
    for (int s = 0; s < L::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < L::BUFS; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 256); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = *tmem_slot;
  // a programmatic dependent of the launch before it: what that wrote is read from here on, through L2 (ld_prev)
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
  const int units = ld_prev(n_tiles) * f_tiles;

  if (warp == 0) {
    if (lane == 0) {
      int i = 0, drawn = 0;
      bool ok = true;
      auto stage_free = [&](int s) { return i < L::STAGES || mbar_wait(&empty[s], (unsigned)((i / L::STAGES - 1) & 1), err, failed, 1); };
      int u = blockIdx.x, after = u < units ? atomicAdd(next, 1) + gridDim.x : units;
      for (; u < units && ok; ++drawn) {
        const int tile = u / f_tiles, f0 = (u - tile * f_tiles) * L::FEATURES;
        const int w0 = ld_prev(tile_expert + tile) * rows_per_expert + f0, w1 = w0 + (L::GATED ? n_out : 128);
        const int x0 = ld_prev(tile_row0 + tile), boxes = (ld_prev(tile_rows + tile) + 63) / 64;
        ring[drawn % L::RING] = u;
        u = after;
        after = u < units ? atomicAdd(next, 1) + gridDim.x : units;      // known long before it is needed
        for (int kb = 0; kb < n_kb; ++kb, ++i) {
          const int s = i % L::STAGES;
          if (!stage_free(s)) { ok = false; break; }
          unsigned char* const at = stages + (size_t)s * L::STAGE_BYTES;
          mbar_expect_tx(&full[s], L::W_BYTES + boxes * 8192);
          tma_load_2d(at, &map_w, kb * 64, w0, &full[s]);
          tma_load_2d(at + L::W_BYTES / 2, &map_w, kb * 64, w1, &full[s]);
          for (int b = 0; b < boxes; ++b) tma_load_2d(at + L::W_BYTES + b * 8192, &map_x, kb * 64, x0 + b * 64, &full[s]);
        }
      }
      if (ok && stage_free(i % L::STAGES)) {
        ring[drawn % L::RING] = -1;
        mbar_arrive(&full[i % L::STAGES]);
        ++i;
      }
      issued_s = i;
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int i = 0;
      bool ok = true;
      for (int done = 0; ok; ++done) {
        ok = mbar_wait(&full[i % L::STAGES], (unsigned)((i / L::STAGES) & 1), err, failed, 3);
        const int b = done % L::BUFS;
        if (ok && done >= L::BUFS) ok = mbar_wait(&acc_empty[b], (unsigned)((done / L::BUFS - 1) & 1), err, failed, 2);
        if (!ok) break;
        const int u = ring[done % L::RING];
        if (u < 0) {
          mbar_arrive(&acc_full[b]);
          break;
        }
        const int n = (ld_prev(tile_rows + u / f_tiles) + 15) / 16 * 16;
        // kind::f16 instruction descriptor: D fp32, A and B bf16, both K-major, N >> 3 at bit 17, M >> 4 at bit 24
        const unsigned id = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((128u >> 4) << 24);
        for (int kb = 0; kb < n_kb; ++kb, ++i) {
          const int s = i % L::STAGES;
          if (kb > 0) ok = mbar_wait(&full[s], (unsigned)((i / L::STAGES) & 1), err, failed, 3);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const unsigned char* const at = stages + (size_t)s * L::STAGE_BYTES;
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const unsigned long long x = umma_desc(at + L::W_BYTES + kk * 32);
            const unsigned acc = kb > 0 || kk > 0 ? 1u : 0u;
            umma(tmem + b * NMAX, umma_desc(at + kk * 32), x, id, acc);
            umma(tmem + 256 + b * NMAX, umma_desc(at + L::W_BYTES / 2 + kk * 32), x, id, acc);
          }
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(&acc_full[b]);
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;      // a quarter of tensor memory's lanes; every other 16 columns
    for (int done = 0;; ++done) {
      const int b = done % L::BUFS;
      const bool ok = mbar_wait(&acc_full[b], (unsigned)((done / L::BUFS) & 1), err, failed, 4);
      if (!__all_sync(0xffffffffu, ok)) break;
      const int u = ring[done % L::RING];
      if (u < 0) break;
      const int tile = u / f_tiles, f0 = (u - tile * f_tiles) * L::FEATURES + q * 32 + lane;
      const int row0 = ld_prev(tile_row0 + tile), rows = ld_prev(tile_rows + tile);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned at = tmem + ((unsigned)(q * 32) << 16) + (unsigned)(b * NMAX);
      for (int c0 = half * 16; c0 < rows; c0 += 32) {
        unsigned r0[16], r1[16];
        tmem_ld16(at + c0, r0);
        tmem_ld16(at + 256 + c0, r1);
        const bool there = c0 + (lane & 15) < rows;       // lane c & 15 looks up what belongs to row c
        const int mine = there && (MODE == 1 || MODE == 3) ? ld_prev(perm + row0 + c0 + (lane & 15)) : 0;
        const float my_w = MODE == 3 && there ? ld_prev(in_w + mine) : 0.f;
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        float v[2][16];
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          float x = __uint_as_float(r0[c]), y = __uint_as_float(r1[c]);
          if (MODE == 0) x = over_one_plus(x, expf(-x)) * y;
          if (MODE == 3) {
            const float sc = __shfl_sync(0xffffffffu, my_w, c);
            const float g = fminf(x * sc, limit), up = fminf(fmaxf(y * sc, -limit), limit);
            x = over_one_plus(g, expf(-alpha * g)) * (up + up_off);
          }
          if (MODE == 2) {
            x = fmaxf(x, 0.f); x *= x;
            y = fmaxf(y, 0.f); y *= y;
          }
          v[0][c] = x;
          v[1][c] = y;
        }
        const int left = rows - c0 - (lane & 1);           // an even lane takes row c of both its and its neighbour's feature, an odd one row c + 1
#pragma unroll
        for (int t = 0; t < (L::GATED ? 1 : 2); ++t) {
          const int f = (f0 + t * 128) & ~1;
          bf16* const to = out + f + (MODE == 1 ? 0 : (size_t)(row0 + c0 + (lane & 1)) * n_out);
          const bool in = f < n_out;
#pragma unroll
          for (int c = 0; c < 16; c += 2) {
            const float got = __shfl_xor_sync(0xffffffffu, lane & 1 ? v[t][c] : v[t][c + 1], 1);
            const unsigned two = lane & 1 ? pack_bf16(got, v[t][c + 1]) : pack_bf16(v[t][c], got);
            if (MODE == 1) {
              const int row = __shfl_sync(0xffffffffu, mine, c + (lane & 1));
              if (c < left && in) *reinterpret_cast<unsigned*>(to + (size_t)row * n_out) = two;
            } else {
              if (c < left && in) *reinterpret_cast<unsigned*>(to + (size_t)c * n_out) = two;
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive(&acc_empty[b]);
    }
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*failed) {   // a wait ran out: give copies and products that may still be in flight a bounded time to end
    const long long t0 = clock64();
    auto expired = [&] { return clock64() - t0 > WAIT_CYCLES; };
    if (threadIdx.x == 0) ring_drain(issued_s, L::STAGES, [&](int s, unsigned parity) { return mbar_try_wait(&full[s], parity); }, expired);
    if (threadIdx.x == 32) {      // the thread that issued the products
      umma_commit(&drained_s);
      while (!mbar_try_wait(&drained_s, 0) && !expired()) {}
    }
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}
// [rows, K] bfloat16 row-major, box 64 k x box_rows rows, 128-byte swizzle, zero fill out of range
bool encode(CUtensorMap* map, const void* base, long long rows, int K, int box_rows) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Sorted { const int *perm, *tile_expert, *tile_row0, *tile_rows, *n_tiles; int* next; int max_tiles; };

template <int MODE, int NMAX>
int tc_launch(const void* x, long long x_rows, const void* w, int E, const Sorted& t, int K, int n_out, void* out, int sms,
              const float* in_w, float limit, float alpha, float up_off, int* err, int pdl, cudaStream_t st) {
  typedef Tc<MODE, NMAX> L;
  CUtensorMap map_w, map_x;
  if (!encode(&map_w, w, (long long)E * (L::GATED ? 2 : 1) * n_out, K, 128) || !encode(&map_x, x, x_rows, K, 64)) return DRYFT_ERR_UNSUPPORTED;
  static std::atomic<unsigned long long> set{0};      // a bit a device (setting the attribute twice does no harm)
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64 || !(set.load(std::memory_order_relaxed) >> dev & 1)) {
    const cudaError_t e = cudaFuncSetAttribute(moe_grouped_tc_kernel<MODE, NMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM);
    if (e != cudaSuccess) return (int)e;
    if (dev < 64) set.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  const int f_tiles = (n_out + L::FEATURES - 1) / L::FEATURES;
  const long long most = (long long)t.max_tiles * f_tiles;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(most < sms ? most : sms));
  cfg.blockDim = dim3(TC_THREADS);
  cfg.dynamicSmemBytes = L::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  const cudaError_t rc = cudaLaunchKernelEx(&cfg, moe_grouped_tc_kernel<MODE, NMAX>, map_w, map_x, t.perm, t.tile_expert, t.tile_row0, t.tile_rows,
                                            t.n_tiles, t.next + (MODE == 1), K / 64, n_out, f_tiles, (bf16*)out, in_w, limit, alpha, up_off, err);
  if (rc != cudaSuccess) return (int)rc;
  return launch_status();
}

// What runs on tcgen05: inner sizes that fill its k slices, and addresses that the copy engine takes.  Many rows of a few very small
// experts are the exception (up to 32 of 128 x 64, more than 1,024 rows: 31 us against 28 on mma.sync, whose small tiles spread over more
// blocks; fewer rows 22 against 27, 64 experts 35 against 38, 256 x 64 as fast).
bool tc_takes(int E, int n_assign, int W, int F, const void* h, const void* w_gate_up, const void* w_down, const void* act, const void* y) {
  const uintptr_t all = (uintptr_t)h | (uintptr_t)w_gate_up | (uintptr_t)w_down | (uintptr_t)act | (uintptr_t)y;
  return W % 64 == 0 && F % 64 == 0 && (all & 15) == 0 && !(E <= 32 && n_assign > 1024 && (long long)W * F <= 128 * 64);
}

// rows per tile: tcgen05: 128 for few rows an expert (accumulators for two units: one is finished while the next is multiplied), 256
// once tiles of 128 would read an expert's weights twice.  Sort, gather and both products, tiles of 128 / 256, 64 experts of 768 x 2,048:
// 112 rows an expert 136 / 152 us, 144 172 / 165, 160 183 / 172, 256 228 / 226, 512 428 / 365; 32 of 512 x 1,024: 112 rows 44 / 45,
// 144 53 / 48, 160 53 / 50, 256 (some experts get more) 70 / 84, 512 90 / 113; 8 of 1,024 x 2,048, one wave of units either way:
// 160 rows 48 / 56, 256 72 / 64, 384 76 / 61, 512 82 / 102.  mma.sync (535, 144 and 127 us of the three at 160
// rows): 128 once an expert gets about a hundred
int tile_rows_for(int n_assign, int E, bool tc) {
  if (tc) return n_assign / E >= 160 ? 256 : 128;
  return n_assign / E >= 96 ? 128 : 64;
}
int max_tiles_for(int n_assign, int E, bool tc) {
  const int bm = tile_rows_for(n_assign, E, tc);
  return (n_assign + bm - 1) / bm + E;
}
}  // namespace

// ints the caller provides in `work`: perm, place [n_assign] | tile_expert, tile_row0, tile_rows [max_tiles] | n_tiles[1] | next[2]
DRYFT_API long long dryft_moe_grouped_work_ints(int n_assign, int E) {
  const int a = max_tiles_for(n_assign, E, true), b = max_tiles_for(n_assign, E, false);
  return 2LL * n_assign + 3LL * (a > b ? a : b) + 3;
}

// y[n*top, C] = experts of idx[n, top] applied to h[n, W]; act [n*top, F] is scratch (sorted order), as y is before its values
// `gated`: 1 = w_gate_up is [E, 2F, W] and the activation is silu(gate) * up; 0 = it is [E, F, W] and the activation is max(., 0)^2;
// 2 = [E, 2F, W] with the clamped activation of MODE 3 (in_w [n*top]: each assignment's weight on the expert's input)
// `pdl`: the tcgen05 products are programmatic dependents of the launches before them; `tcgen05` 0: the mma.sync products at any size
DRYFT_API int dryft_moe_grouped(const void* h, const void* w_gate_up, const void* w_down, const int* idx, int n_tokens, int top,
                                int E, int W, int F, void* act, void* y, int* work, int gated, const float* in_w, float limit,
                                float alpha, float up_off, int* err, int pdl, int tcgen05, cudaStream_t st) {
  if (n_tokens <= 0) return 0;
  if (top < 1 || E < 1 || W % 16 || F % 16 || W < 16 || F < 16 || gated < 0 || gated > 2 || (gated == 2 && !in_w)) return DRYFT_ERR_UNSUPPORTED;
  const long long n_assign_ll = (long long)n_tokens * top;
  if (n_assign_ll > (1LL << 30) || (size_t)E * 2 * sizeof(int) > 48 * 1024 || (long long)E * 2 * F > (1LL << 31) - 1 ||
      (long long)E * W > (1LL << 31) - 1)
    return DRYFT_ERR_UNSUPPORTED;
  const int n_assign = (int)n_assign_ll;
  const bool tc = tcgen05 && tc_takes(E, n_assign, W, F, h, w_gate_up, w_down, act, y);
  const int bm = tile_rows_for(n_assign, E, tc), max_tiles = max_tiles_for(n_assign, E, tc);
  int* const perm = work;
  int* const place = perm + n_assign;
  int* const tile_expert = place + n_assign;
  int* const tile_row0 = tile_expert + max_tiles;
  int* const tile_rows = tile_row0 + max_tiles;
  int* const n_tiles = tile_rows + max_tiles;
  int hists = SORT_INTS / E - 1;
  hists = hists > SORT_THREADS / 32 ? SORT_THREADS / 32 : hists;
  if (hists > n_assign / 256) hists = n_assign / 256;      // few assignments hardly collide: less to clear and to add up
  if (hists < 1) hists = 1;
  moe_sort_kernel<<<1, SORT_THREADS, sizeof(int) * (hists + 1) * E, st>>>(idx, n_assign, E, bm, hists, perm, tc ? place : nullptr,
                                                                                  tile_expert, tile_row0, tile_rows, n_tiles, n_tiles + 1);
  int rc = launch_status();
  if (rc) return rc;
  if (tc) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const Sorted t = {perm, tile_expert, tile_row0, tile_rows, n_tiles, n_tiles + 1, max_tiles};
    const int gather_blocks = (n_assign + 7) / 8;
    (gather_blocks <= SIGNAL_BLOCKS ? moe_gather_kernel<true> : moe_gather_kernel<false>)<<<gather_blocks, 256, 0, st>>>(
        (const uint4*)h, place, n_assign, top, W / 8, (uint4*)y, perm);
    rc = launch_status();
    if (rc) return rc;
    auto both = [&](auto nmax) {
      constexpr int N = decltype(nmax)::value;
      int r = gated == 2 ? tc_launch<3, N>(y, n_assign, w_gate_up, E, t, W, F, act, sms, in_w, limit, alpha, up_off, err, pdl, st)
              : gated    ? tc_launch<0, N>(y, n_assign, w_gate_up, E, t, W, F, act, sms, nullptr, 0.f, 1.f, 0.f, err, pdl, st)
                         : tc_launch<2, N>(y, n_assign, w_gate_up, E, t, W, F, act, sms, nullptr, 0.f, 1.f, 0.f, err, pdl, st);
      return r ? r : tc_launch<1, N>(act, n_assign, w_down, E, t, F, W, y, sms, nullptr, 0.f, 1.f, 0.f, err, pdl, st);
    };
    return bm == 256 ? both(std::integral_constant<int, 256>()) : both(std::integral_constant<int, 128>());
  }
  auto both = [&](auto rows) {
    constexpr int BM = decltype(rows)::value;
    int r = gated == 2 ? gemm_launch<3, BM, 64>(h, w_gate_up, perm, tile_expert, tile_row0, tile_rows, n_tiles, top, W, F, act, max_tiles, st,
                                                in_w, limit, alpha, up_off)
            : gated    ? gemm_launch<0, BM, 64>(h, w_gate_up, perm, tile_expert, tile_row0, tile_rows, n_tiles, top, W, F, act, max_tiles, st)
                       : gemm_launch<2, BM, 64>(h, w_gate_up, perm, tile_expert, tile_row0, tile_rows, n_tiles, top, W, F, act, max_tiles, st);
    return r ? r : gemm_launch<1, BM, 128>(act, w_down, perm, tile_expert, tile_row0, tile_rows, n_tiles, top, F, W, y, max_tiles, st);
  };
  return bm == 128 ? both(std::integral_constant<int, 128>()) : both(std::integral_constant<int, 64>());
}
