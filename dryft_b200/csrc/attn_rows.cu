// Attention of independent query rows over the paged cache ("split-KV"): the decode kernel of both
// precisions, and the prefill kernel of the 32-bit path (a prompt token is just a row with its own
// position).  Compiled per model with -DDRYFT_HEAD_DIM, -DDRYFT_GROUP, -DDRYFT_PAGE.
//
// Grid (rows, kv heads, splits).  One block serves the GROUP query heads that share a kv head for
// one query row over one contiguous range of keys.  Row n at position p of slot s sees the
// keys j with  max(0, p+1-window) <= j <= p  (window <= 0: all keys) — the new token's own key is
// already in the cache (hari495/dryft, engine/dryft_qwen3/model.py:235,249-257;
// kernels/attn_decode.py:8-10,52-55).  Scores, the running maximum and the sums are 32-bit
// (attn_decode.py:77-90).  With one split the block writes the output; otherwise it writes an
// un-normalised partial (acc, m, l) and `attn_rows_reduce_kernel` combines them
// (attn_decode.py:102-118).
//
// A split is 16 keys, half a page or whole pages: a block takes 10 us for the 64 keys of a page (32-bit, two trips to memory, scores and
// values of 64 keys by 128 threads), and while rows are few most blocks of a launch would have none.  Four rows of about 150 keys, two kv
// heads, 32 splits: 11 + 5.5 us for the two launches by pages, 6.0 + 4.3 by 16 keys.
//
// No block waits on another block; there is no spin anywhere in this file.
#include "common.cuh"
#include "attn_rows_static.h"
#include <math.h>
#include <type_traits>

#if !defined(DRYFT_HEAD_DIM) || !defined(DRYFT_GROUP) || !defined(DRYFT_PAGE)
#error "compile with -DDRYFT_HEAD_DIM=.. -DDRYFT_GROUP=.. -DDRYFT_PAGE=.."
#endif

namespace {
constexpr int D = DRYFT_HEAD_DIM;
constexpr int G = DRYFT_GROUP;
constexpr int PAGE = DRYFT_PAGE;
constexpr int GRAIN = 16;
constexpr int THREADS = 128;
constexpr int NWARP = THREADS / 32;
constexpr int DIMS_PER_THREAD = (D + THREADS - 1) / THREADS;
static_assert(D % 16 == 0, "head size must be a multiple of 16");
static_assert(PAGE % 32 == 0, "page size must be a multiple of 32");

template <typename T> struct Smem {
  static constexpr int VEC = 16 / sizeof(T);       // elements per 16-byte vector
  static constexpr int KSTRIDE = D + VEC;          // padded K row: conflict-free row-per-thread reads
  static constexpr size_t bytes() {
    return sizeof(float) * (G * D + G * PAGE + 3 * G) + sizeof(T) * (size_t)(PAGE * KSTRIDE + PAGE * D) + 32;
  }
  // Blocks a multiprocessor that the registers have to leave room for: as many as shared memory does, up to what costs few spills.  16 heads on one
  // kv head, 1,500 rows of 800 keys, us with room for 5 / 7: 32 dims, 32-bit 287 / 259, bfloat16 268 / 222, 64 dims, bfloat16 385 / 352.
  static constexpr int blocks() {
    const size_t n = 227 * 1024 / (bytes() + 1024), most = G > 8 ? 7 : G > 2 ? 8 : 10;
    return n < 1 ? 1 : (int)(n > most ? most : n);
  }
};

template <typename T>
__global__ void __launch_bounds__(THREADS, Smem<T>::blocks()) attn_rows_kernel(
    const T* __restrict__ q,                                   // [N, nH, D]
    const T* __restrict__ k_pages, const T* __restrict__ v_pages,  // [pages, nKV, PAGE, D]
    const int* __restrict__ page_table, int max_pages,
    const int* __restrict__ tok_slot, const int* __restrict__ tok_pos,
    T* __restrict__ out,                                       // [N, nH*D]
    float* __restrict__ part_o, float* __restrict__ part_ml,   // [N, nH, S, D], [N, nH, S, 2]
    int nKV, int n_splits, float scale, int window) {
  let_next_launch_in();   // a product behind this launch may start on its weights
  using L = Smem<T>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* kt = reinterpret_cast<T*>(smem_raw);                 // [PAGE][KSTRIDE]
  T* vt = kt + PAGE * L::KSTRIDE;                         // [PAGE][D]
  float* qs = reinterpret_cast<float*>(vt + PAGE * D);    // [G][D]
  float* sc = qs + G * D;                                 // [G][PAGE]
  float* m_s = sc + G * PAGE;                             // [G]
  float* l_s = m_s + G;
  float* a_s = l_s + G;

  const int n = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int nH = nKV * G;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int slot = tok_slot[n];

  if (slot < 0) {  // padding row: defined zeros, no cache access
    if (n_splits == 1) {
      for (int i = tid; i < G * D; i += THREADS) out[(size_t)n * nH * D + (size_t)kvh * G * D + i] = from_f32<T>(0.f);
    } else {
      for (int g = 0; g < G; ++g) {
        size_t pi = ((size_t)n * nH + kvh * G + g) * n_splits + split;
        for (int d = tid; d < D; d += THREADS) part_o[pi * D + d] = 0.f;
        if (tid == 0) { part_ml[pi * 2] = -INFINITY; part_ml[pi * 2 + 1] = 0.f; }
      }
    }
    return;
  }

  const int pos = tok_pos[n];
  const int kv_hi = pos + 1;                                        // exclusive
  const int kv_lo = window > 0 ? max(0, kv_hi - window) : 0;        // inclusive
  constexpr int PAGE_GRAINS = PAGE / GRAIN;
  const int base = kv_lo / PAGE * PAGE, grains = (kv_hi - base + GRAIN - 1) / GRAIN;
  int per_split = (grains + n_splits - 1) / n_splits;
  if (per_split > PAGE_GRAINS / 2) per_split = (per_split + PAGE_GRAINS - 1) / PAGE_GRAINS * PAGE_GRAINS;      // no page in more parts than needed
  const int k_begin = max(kv_lo, (int)min((long long)base + (long long)split * per_split * GRAIN, (long long)kv_hi));      // this block's keys
  const int k_end = (int)min((long long)base + (long long)(split + 1) * per_split * GRAIN, (long long)kv_hi);
  if (n_splits > 1 && k_begin >= k_end) {      // nothing to add: a maximum of -inf says so
    if (tid < G) {
      const size_t pi = ((size_t)n * nH + kvh * G + tid) * n_splits + split;
      part_ml[pi * 2] = -INFINITY;
      part_ml[pi * 2 + 1] = 0.f;
    }
    return;
  }

  for (int i = tid; i < G * D; i += THREADS) qs[i] = to_f32<T>(q[((size_t)n * nH + (size_t)kvh * G) * D + i]);
  if (tid < G) { m_s[tid] = -INFINITY; l_s[tid] = 0.f; a_s[tid] = 1.f; }
  float acc[DIMS_PER_THREAD][G];
#pragma unroll
  for (int i = 0; i < DIMS_PER_THREAD; ++i)
#pragma unroll
    for (int g = 0; g < G; ++g) acc[i][g] = 0.f;

  const int* pt = page_table + (size_t)slot * max_pages;
  constexpr int VPR = D / L::VEC;  // 16-byte vectors per row
  // One page, of whose keys rows [r0, r1) are this block's.  `whole`: it is walked from end to end with constant bounds, zeros and probabilities of
  // zero beside the block's own; else only the groups of eight rows that hold some of them are.  With bounds that only the launch knows, launches
  // of many rows were up to 1.37 times as long: probabilities read one by one instead of four at a time, a division an item, registers for
  // loads that no thread makes.
  auto walk = [&](auto whole, int pg) {
    constexpr bool WHOLE = decltype(whole)::value;
    const int page = pt[pg];
    const int p0 = pg * PAGE;
    const int r0 = max(k_begin - p0, 0), r1 = min(k_end - p0, PAGE);
    const int ra = WHOLE ? 0 : r0 & ~7, rb = WHOLE ? PAGE : (r1 + 7) & ~7, rows = rb - ra;
    const T* kp = k_pages + ((size_t)page * nKV + kvh) * PAGE * D;
    const T* vp = v_pages + ((size_t)page * nKV + kvh) * PAGE * D;
    __syncthreads();  // previous tile fully consumed
    // words of K and of V on their way at once: eight of a whole page (two at a time left it eight trips to memory long), else two grains'
    constexpr int GRAINS = 2 * GRAIN * VPR / THREADS, AHEAD = WHOLE || GRAINS > 8 ? 8 : GRAINS < 2 ? 2 : GRAINS;
    for (int i0 = ra * VPR + tid; i0 < rb * VPR; i0 += AHEAD * THREADS) {
      uint4 kv4[AHEAD], vv4[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int i = i0 + u * THREADS, r = i / VPR, c = i % VPR;
        kv4[u] = vv4[u] = make_uint4(0, 0, 0, 0);
        if (i < rb * VPR && r >= r0 && r < r1) {
          kv4[u] = reinterpret_cast<const uint4*>(kp + (size_t)r * D)[c];
          vv4[u] = reinterpret_cast<const uint4*>(vp + (size_t)r * D)[c];
        }
      }
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int i = i0 + u * THREADS, r = i / VPR, c = i % VPR;
        if (i < rb * VPR) {
          *reinterpret_cast<uint4*>(kt + r * L::KSTRIDE + c * L::VEC) = kv4[u];
          *reinterpret_cast<uint4*>(vt + r * D + c * L::VEC) = vv4[u];
        }
      }
    }
    __syncthreads();
    // scores: item -> (head g, key r); consecutive threads take consecutive keys, or two or four threads one key where the items are few (not
    // of a whole page: the threads of a key read the same banks)
    const int items = G * rows, share = WHOLE || 2 * items > THREADS ? 1 : 4 * items > THREADS ? 2 : 4;
    for (int i0 = 0; i0 < items * share; i0 += THREADS) {
      const int item = (i0 + tid) / share, sub = tid % share;
      const int g = item / rows, r = ra + item - g * rows;
      const bool seen = item < items && r >= r0 && r < r1;
      float dot[4] = {0.f, 0.f, 0.f, 0.f};      // four chains of D / 4: one of D waits for every addition
      if (seen) {
        const T* kr = kt + r * L::KSTRIDE;
        const float* qg = qs + g * D;
#pragma unroll 4
        for (int c = sub; c < VPR; c += share) {
          uint4 raw = *reinterpret_cast<const uint4*>(kr + c * L::VEC);
          const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int t = 0; t < L::VEC; t += 4) {
            const float4 q4 = *reinterpret_cast<const float4*>(qg + c * L::VEC + t);
            dot[0] = fmaf(q4.x, to_f32<T>(e[t]), dot[0]);
            dot[1] = fmaf(q4.y, to_f32<T>(e[t + 1]), dot[1]);
            dot[2] = fmaf(q4.z, to_f32<T>(e[t + 2]), dot[2]);
            dot[3] = fmaf(q4.w, to_f32<T>(e[t + 3]), dot[3]);
          }
        }
      }
      float s = (dot[0] + dot[1]) + (dot[2] + dot[3]);
      for (int o = 1; o < share; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (item < items && sub == 0) sc[g * PAGE + r] = seen ? s * scale : -INFINITY;
    }
    __syncthreads();
    // online softmax, one warp per head
    for (int g = warp; g < G; g += NWARP) {
      float mx = -INFINITY;
      for (int r = ra + lane; r < rb; r += 32) mx = fmaxf(mx, sc[g * PAGE + r]);
      mx = warp_max(mx);
      const float m_old = m_s[g];
      const float m_new = fmaxf(m_old, mx);
      float sum = 0.f;
      for (int r = ra + lane; r < rb; r += 32) {
        const float s = sc[g * PAGE + r];
        const float p = (s == -INFINITY) ? 0.f : expf(s - m_new);
        sc[g * PAGE + r] = p;
        sum += p;
      }
      sum = warp_sum(sum);
      if (lane == 0) {
        const float alpha = (m_old == -INFINITY) ? 0.f : expf(m_old - m_new);
        a_s[g] = alpha;
        m_s[g] = m_new;
        l_s[g] = l_s[g] * alpha + sum;
      }
    }
    __syncthreads();
    // acc = acc*alpha + P V ; thread owns output dims tid, tid+THREADS, ...
#pragma unroll
    for (int i = 0; i < DIMS_PER_THREAD; ++i) {
      const int d = tid + i * THREADS;
      if (d < D) {
#pragma unroll
        for (int g = 0; g < G; ++g) acc[i][g] *= a_s[g];
        for (int r = ra; r < rb; r += 8) {
          float v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) v[u] = to_f32<T>(vt[(r + u) * D + d]);
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int u = 0; u < 8; u += 4) {
              const float4 p = *reinterpret_cast<const float4*>(sc + g * PAGE + r + u);
              acc[i][g] = fmaf(p.x, v[u], acc[i][g]);
              acc[i][g] = fmaf(p.y, v[u + 1], acc[i][g]);
              acc[i][g] = fmaf(p.z, v[u + 2], acc[i][g]);
              acc[i][g] = fmaf(p.w, v[u + 3], acc[i][g]);
            }
        }
      }
    }
  };
  // More than half a page of keys is walked as a whole one: 64 rows of 300 keys (the last page has 44), 8 heads of 64 in bfloat16, us as a
  // part / as a whole page: one split 13.0 / 12.1, four 13.9 / 12.6.  A few keys are not: 200 rows of 130, 32-bit, 8 heads of 64 on four 13.8 / 14.6.
  for (int pg = k_begin / PAGE; pg * PAGE < k_end; ++pg) {
    if (min(k_end, (pg + 1) * PAGE) - max(k_begin, pg * PAGE) > PAGE / 2) walk(std::true_type{}, pg);
    else walk(std::false_type{}, pg);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < DIMS_PER_THREAD; ++i) {
    const int d = tid + i * THREADS;
    if (d >= D) continue;
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int h = kvh * G + g;
      if (n_splits == 1) {
        const float l = l_s[g];
        out[((size_t)n * nH + h) * D + d] = from_f32<T>(l > 0.f ? acc[i][g] / l : 0.f);
      } else {
        part_o[(((size_t)n * nH + h) * n_splits + split) * D + d] = acc[i][g];
      }
    }
  }
  if (n_splits > 1 && tid < G) {
    size_t pi = ((size_t)n * nH + kvh * G + tid) * n_splits + split;
    part_ml[pi * 2] = m_s[tid];
    part_ml[pi * 2 + 1] = l_s[tid];
  }
}

// Combine the partials of one (row, head):  w_s = exp(m_s - max m);  o = sum w_s acc_s / sum w_s l_s, in the order of the splits.  A thread
// makes the weights of some splits, all of them share them; sixteen splits' values are on their way together at up to 128 dims,
// eight above.
constexpr int REDUCE_TILE = 128;
constexpr int REDUCE_THREADS = D < 128 ? 64 : 128;
template <typename T>
__global__ void __launch_bounds__(REDUCE_THREADS) attn_rows_reduce_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                               T* __restrict__ out, int n_splits) {
  let_next_launch_in();   // a product behind this launch may start on its weights
  __shared__ float wgt[REDUCE_TILE], sum[REDUCE_TILE], top[REDUCE_THREADS / 32];
  const size_t rh = blockIdx.x;  // row * nH + head
  const float* ml = part_ml + rh * n_splits * 2;
  const int tid = threadIdx.x;
  float mx = -INFINITY;
  for (int s = tid; s < n_splits; s += REDUCE_THREADS) mx = fmaxf(mx, ml[s * 2]);
  mx = warp_max(mx);
  if (tid % 32 == 0) top[tid / 32] = mx;
  __syncthreads();
  mx = top[0];
  for (int w = 1; w < REDUCE_THREADS / 32; ++w) mx = fmaxf(mx, top[w]);
  constexpr int MINE = (D + REDUCE_THREADS - 1) / REDUCE_THREADS;      // dims a thread
  float num[MINE], denom = 0.f;
#pragma unroll
  for (int i = 0; i < MINE; ++i) num[i] = 0.f;
  for (int s0 = 0; s0 < n_splits; s0 += REDUCE_TILE) {
    const int n = min(REDUCE_TILE, n_splits - s0);
    for (int s = tid; s < n; s += REDUCE_THREADS) {
      const float m = ml[(s0 + s) * 2];
      wgt[s] = m == -INFINITY ? -1.f : expf(m - mx);      // -1: an empty split, which wrote no values
      sum[s] = ml[(s0 + s) * 2 + 1];
    }
    __syncthreads();
    constexpr int AT_ONCE = 16 / MINE;
    for (int q = 0; q < n; q += AT_ONCE) {
      float v[AT_ONCE][MINE];
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u)
#pragma unroll
        for (int i = 0; i < MINE; ++i) {
          const int d = tid + i * REDUCE_THREADS;
          v[u][i] = q + u < n && d < D ? part_o[(rh * n_splits + s0 + q + u) * D + d] : 0.f;
        }
#pragma unroll
      for (int u = 0; u < AT_ONCE; ++u) {
        if (q + u >= n || wgt[q + u] == -1.f) continue;
        denom += wgt[q + u] * sum[q + u];
#pragma unroll
        for (int i = 0; i < MINE; ++i) num[i] += wgt[q + u] * v[u][i];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < MINE; ++i) {
    const int d = tid + i * REDUCE_THREADS;
    if (d < D) out[rh * D + d] = from_f32<T>(denom > 0.f ? num[i] / denom : 0.f);
  }
}

template <typename T>
int launch(const void* q, const void* k_pages, const void* v_pages, const int* page_table, int max_pages,
           const int* tok_slot, const int* tok_pos, void* out, float* part_o, float* part_ml, int n_rows, int nKV,
           int n_splits, float scale, int window, cudaStream_t st) {
  if (n_rows <= 0) return 0;
  if (n_splits < 1 || nKV < 1 || nKV > 65535 || n_splits > 65535) return DRYFT_ERR_UNSUPPORTED;
  if (n_splits > 1 && (!part_o || !part_ml)) return DRYFT_ERR_UNSUPPORTED;
  const size_t smem = Smem<T>::bytes();
  if (smem > 227 * 1024) return DRYFT_ERR_UNSUPPORTED;
  // per instantiation and per device (the attribute belongs to the device's copy of the kernel); set outside any
  // stream capture by the first (eager) launch on that device
  static bool attr_set[64] = {false};
  if (smem > 48 * 1024) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return (int)e;
    if (dev < 0 || dev >= 64) return DRYFT_ERR_UNSUPPORTED;
    if (!attr_set[dev]) {
      e = cudaFuncSetAttribute(attn_rows_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return (int)e;
      attr_set[dev] = true;
    }
  }
  dim3 grid(n_rows, nKV, n_splits);
  attn_rows_kernel<T><<<grid, THREADS, smem, st>>>((const T*)q, (const T*)k_pages, (const T*)v_pages, page_table,
                                                  max_pages, tok_slot, tok_pos, (T*)out, part_o, part_ml, nKV,
                                                  n_splits, scale, window);
  int rc = launch_status();
  if (rc || n_splits == 1) return rc;
  attn_rows_reduce_kernel<T><<<(unsigned)((size_t)n_rows * nKV * G), REDUCE_THREADS, 0, st>>>(part_o, part_ml, (T*)out, n_splits);
  return launch_status();
}
}  // namespace

// The sizes this library was compiled for; the loader checks them against the model's.
DRYFT_API int dryft_attn_rows_head_dim() { return D; }
DRYFT_API int dryft_attn_rows_group() { return G; }
DRYFT_API int dryft_attn_rows_page() { return PAGE; }

DRYFT_API int dryft_attn_rows(int is_bf16, const void* q, const void* k_pages, const void* v_pages, const int* page_table,
                              int max_pages, const int* tok_slot, const int* tok_pos, void* out, float* part_o,
                              float* part_ml, int n_rows, int nKV, int n_splits, float scale, int window, cudaStream_t st) {
  return is_bf16 ? launch<__nv_bfloat16>(q, k_pages, v_pages, page_table, max_pages, tok_slot, tok_pos, out, part_o, part_ml,
                                         n_rows, nKV, n_splits, scale, window, st)
                 : launch<float>(q, k_pages, v_pages, page_table, max_pages, tok_slot, tok_pos, out, part_o, part_ml,
                                 n_rows, nKV, n_splits, scale, window, st);
}

// ------------------------------------------------------------------------------------------
// The same attention for callers that cannot allocate device memory (see attn_rows_static.h).
// The split partials live in a file-scope device array instead of buffers handed in.  In host
// code the array's name is only a stand-in for the symbol, not a device address, so the address
// is asked of the runtime once per device, with that device current, and kept.
// ------------------------------------------------------------------------------------------
namespace {
static __device__ __align__(256) float g_static_scratch[DRYFT_ATTN_ROWS_STATIC_FLOATS];
constexpr int MAX_DEVICES = 64;
float* g_static_scratch_ptr[MAX_DEVICES] = {nullptr};
}  // namespace

DRYFT_API int dryft_attn_rows_static_scratch(int is_bf16, const void* q, const void* k_pages, const void* v_pages,
                                             const int* page_table, int max_pages, const int* tok_slot, const int* tok_pos,
                                             void* out, int n_rows, int nKV, int n_splits, float scale, int window,
                                             cudaStream_t st) {
  if (n_rows <= 0) return 0;
  if (n_splits < 1 || nKV < 1 || nKV > 65535 || n_splits > 65535) return DRYFT_ERR_UNSUPPORTED;  // the grid's limits
  // partial outputs [rows, heads, splits, D] and (max, sum) pairs [rows, heads, splits, 2].  The size check divides
  // instead of multiplying, so that no count, however large, can wrap around and pass.
  const unsigned long long heads = (unsigned long long)nKV * G;                      // < 2^20
  const unsigned long long per_row = heads * (unsigned long long)n_splits * (D + 2);  // < 2^45
  if (n_splits > 1 && (unsigned long long)n_rows > (unsigned long long)DRYFT_ATTN_ROWS_STATIC_FLOATS / per_row)
    return DRYFT_ERR_SCRATCH_TOO_SMALL;
  const unsigned long long need_o = (unsigned long long)n_rows * heads * n_splits * D;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= MAX_DEVICES) return DRYFT_ERR_UNSUPPORTED;
  if (g_static_scratch_ptr[dev] == nullptr) {  // set-up, once per device: the first call on a device
    float* ptr = nullptr;
    e = cudaGetSymbolAddress((void**)&ptr, g_static_scratch);
    if (e != cudaSuccess) return (int)e;
    g_static_scratch_ptr[dev] = ptr;
  }
  float* part_o = g_static_scratch_ptr[dev];
  float* part_ml = part_o + need_o;
  // Nothing in the scratch has to start at zero: every split writes its maximum and sum of every
  // (row, head), and its values where it had keys, before the combining kernel reads any of them.
  return is_bf16 ? launch<__nv_bfloat16>(q, k_pages, v_pages, page_table, max_pages, tok_slot, tok_pos, out, part_o, part_ml,
                                         n_rows, nKV, n_splits, scale, window, st)
                 : launch<float>(q, k_pages, v_pages, page_table, max_pages, tok_slot, tok_pos, out, part_o, part_ml,
                                 n_rows, nKV, n_splits, scale, window, st);
}

DRYFT_API long long dryft_attn_rows_static_scratch_floats() { return (long long)DRYFT_ATTN_ROWS_STATIC_FLOATS; }
