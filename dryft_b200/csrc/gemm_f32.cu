// True 32-bit matrix product  C[M,N] = A[M,K] * W[N,K]^T  on the CUDA cores: fp32 operands,
// fp32 fused multiply-adds, no tensor-core (TF32) mode.  It stands where hari495/dryft calls
// F.linear with TF32 switched off (engine/engine.py:32-33; engine/dryft_qwen3/model.py:153),
// and is the matrix product of the library's 32-bit path.
//
// One order of additions for every inner size: up to K = 256 one chain in order; beyond it k is cut into chunks of 64, a chunk is
// accumulated in order from zero by one thread, and the chunks' sums are added in order.  So a row's result does not depend on
// how many other rows are in the batch or on which of the kernels below ran: in the 32-bit path the same token gives bit-identical
// projections whether it is run alone, in a prompt or in a batch.  (The order lets few rows spread k over threads, and
// is closer to the exact sum than one chain of K additions: 1.7e-7 against 5.6e-7 at K = 1,030, 2.8e-7 against 1.8e-6 at
// K = 9,728.)
// Any M, N, K >= 1; lda/ldc are row strides in elements.
#include "common.cuh"

namespace {
constexpr int CH = 64;        // k per chunk
// Inner sizes up to this are one chunk, of the tiles: they keep the order of one chain, the only one that small models' sums have had.
// That costs them closeness (K = 256: 2.9e-7 off 64 bits; chunks 1.5e-7, at every size) and few rows the kernel that streams (1 row
// and 1,024 outputs over 64 / 128 / 256: 3.9 / 6.5 / 11.6 us; streamed 1.7 / 1.9 / 1.9; 64 rows and 4,096 outputs alike).
constexpr int ONE_CHAIN = 256;
constexpr int CHP = CH + 4;   // a chunk of activations in shared memory: chunks start in different banks

template <int VEC> __device__ __forceinline__ void copy_async(float* dst, const float* src, bool there) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = there ? 4 * VEC : 0;   // nothing read, zeros written
  if (VEC == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---------------------------------------------------------------------------- few rows
// Bound by the weights' bytes.  A block streams pieces of W -- R rows x 256/R chunks, 64 KB -- through two or three stages
// of shared memory by asynchronous copies; a thread owns one chunk of two of the piece's rows and 2 MT sums, so that a
// broadcast of activations serves two rows (with one row a thread those reads were the bound).  16-byte words of W are
// swizzled by their reader's lane: eight lanes read eight different bank groups.  R: long rows are cut among more threads
// (8 rows x 2,048 k, 16 x 1,024, 32 x 512), so that few outputs still fill the SMs.  XRES: all of A's rows stay in shared
// memory; otherwise a piece brings its own columns of A.
template <int MT, int R, int VEC, bool XRES, int STAGES>
__global__ void __launch_bounds__(128) gemm_f32_few_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W,
                                                           float* __restrict__ C, int ldc, int M, int N, int K, int x_chunks) {
  constexpr int Q = 256 / R, KP = Q * CH, H = R / 2;
  constexpr int OUTS = (R * MT + 127) / 128;
  A += (size_t)blockIdx.y * MT * lda;      // a row of blocks for each MT rows
  C += (size_t)blockIdx.y * MT * ldc;
  M -= (int)blockIdx.y * MT;
  extern __shared__ float4 smem4[];
  float* const wst = reinterpret_cast<float*>(smem4);             // [STAGES][R][KP]
  float* const part = wst + STAGES * R * KP;                      // [MT][Q][R]
  float* const xs = part + MT * Q * R;                            // [XRES ? 1 : STAGES][MT][x_chunks][CHP]
  const int tid = threadIdx.x, r = tid % H, q = tid / H;
  const int tiles = (N + R - 1) / R, pieces = (K + KP - 1) / KP;
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int steps = mine * pieces;

  auto load_x = [&](float* to, int k0, int chunks) {
    const int per = chunks * (CH / VEC);
    for (int i = tid; i < MT * per; i += 128) {
      const int m = i / per, c = (i % per) * VEC, k = k0 + c;
      const bool there = m < M && k < K;
      copy_async<VEC>(to + ((size_t)m * x_chunks + c / CH) * CHP + c % CH, there ? A + (size_t)m * lda + k : A, there);
    }
  };
  auto load_w = [&](int step) {
    if (step < steps) {
      const int n0 = ((int)blockIdx.x + (step / pieces) * (int)gridDim.x) * R, k0 = (step % pieces) * KP;
      float* const to = wst + (step % STAGES) * R * KP;
#pragma unroll 4
      for (int i = tid; i < R * KP / VEC; i += 128) {
        const int row = i / (KP / VEC), c = (i % (KP / VEC)) * VEC;
        const int swz = (row % H + H * (c / CH)) & 7;
        const bool there = n0 + row < N && k0 + c < K;
        copy_async<VEC>(to + row * KP + (c ^ (swz * 4)), there ? W + (size_t)(n0 + row) * K + k0 + c : W, there);
      }
    }
  };
  auto load_own_x = [&](int step) {
    if (!XRES && step < steps) load_x(xs + (size_t)(step % STAGES) * MT * x_chunks * CHP, (step % pieces) * KP, Q);
  };
  // the first weights depend on nothing; the activations are the launch before's (a programmatic dependent: 16-byte copies only,
  // which go past L1)
#pragma unroll
  for (int s = 0; s < STAGES; ++s) load_w(s);
  asm volatile("griddepcontrol.launch_dependents;\n\tgriddepcontrol.wait;" ::: "memory");
  if (XRES) load_x(xs, 0, x_chunks);
#pragma unroll
  for (int s = 0; s < STAGES; ++s) load_own_x(s);
#pragma unroll
  for (int s = 0; s < STAGES; ++s) copies_commit();      // everything so far is the first group's
  float total[OUTS];
  for (int s = 0; s < steps; ++s) {
    const int p = s % pieces;
    copies_wait<STAGES - 1>();
    __syncthreads();
    const float* w = wst + (s % STAGES) * R * KP + r * KP + q * CH;
    const int xc = XRES ? p * Q + q : q;
    const float* x = xs + (XRES ? 0 : (size_t)(s % STAGES) * MT * x_chunks * CHP) + (size_t)xc * CHP;
    float acc[2][MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[0][m] = acc[1][m] = 0.f;
    if (!XRES || xc < x_chunks) {
#pragma unroll(MT <= 4 ? 8 : 2)
      for (int i = 0; i < CH; i += 4) {
        const float4 w0 = *reinterpret_cast<const float4*>(w + (i ^ ((tid & 7) * 4)));
        const float4 w1 = *reinterpret_cast<const float4*>(w + H * KP + (i ^ ((tid & 7) * 4)));
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const float4 xv = *reinterpret_cast<const float4*>(x + (size_t)m * x_chunks * CHP + i);
          acc[0][m] = fmaf(xv.w, w0.w, fmaf(xv.z, w0.z, fmaf(xv.y, w0.y, fmaf(xv.x, w0.x, acc[0][m]))));
          acc[1][m] = fmaf(xv.w, w1.w, fmaf(xv.z, w1.z, fmaf(xv.y, w1.y, fmaf(xv.x, w1.x, acc[1][m]))));
        }
      }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      part[(m * Q + q) * R + r] = acc[0][m];
      part[(m * Q + q) * R + H + r] = acc[1][m];
    }
    __syncthreads();
    load_w(s + STAGES);    // into the stage that every thread has just left
    load_own_x(s + STAGES);
    copies_commit();
    const int n0 = ((int)blockIdx.x + (s / pieces) * (int)gridDim.x) * R;
#pragma unroll
    for (int o = 0; o < OUTS; ++o) {
      const int i = tid + o * 128;
      if (R * MT % 128 != 0 && i >= R * MT) continue;
      const int m = i / R, row = i % R;
      float t = p == 0 ? 0.f : total[o];
#pragma unroll
      for (int c = 0; c < Q; ++c) t += part[(m * Q + c) * R + row];
      total[o] = t;
      if (p == pieces - 1 && m < M && n0 + row < N) C[(size_t)m * ldc + n0 + row] = t;
    }
  }
  copies_wait<0>();
}

template <int MT, int R, int VEC, bool XRES, int STAGES>
int launch_few(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K, int x_chunks, size_t smem, int sms, int pdl,
               cudaStream_t st) {
  auto kern = gemm_f32_few_kernel<MT, R, VEC, XRES, STAGES>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int tiles = (N + R - 1) / R;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles < sms ? tiles : sms, (M + MT - 1) / MT);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl && VEC == 4 ? 1 : 0;
  e = cudaLaunchKernelEx(&cfg, kern, A, lda, W, C, ldc, M, N, K, x_chunks);
  return e != cudaSuccess ? (int)e : launch_status();
}

template <int MT, int R, int VEC>
int launch_few_x(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K, int sms, int pdl, cudaStream_t st) {
  constexpr int Q = 256 / R;
  constexpr size_t most = 227 * 1024, stage = 64 * 1024, part = (size_t)4 * MT * 256;
  static_assert(2 * (stage + (size_t)4 * MT * Q * CHP) + part <= most, "two stages with their own columns of A fit a block");
  const int all = (K + CH - 1) / CH;
  const size_t x = (size_t)4 * MT * all * CHP;
  if (3 * stage + part + x <= most) return launch_few<MT, R, VEC, true, 3>(A, lda, W, C, ldc, M, N, K, all, 3 * stage + part + x, sms, pdl, st);
  if (2 * stage + part + x <= most) return launch_few<MT, R, VEC, true, 2>(A, lda, W, C, ldc, M, N, K, all, 2 * stage + part + x, sms, pdl, st);
  return launch_few<MT, R, VEC, false, 2>(A, lda, W, C, ldc, M, N, K, Q, 2 * (stage + (size_t)4 * MT * Q * CHP) + part, sms, pdl, st);
}

template <int MT, int VEC>
int launch_few_r(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K, int sms, int pdl, cudaStream_t st) {
  // the more rows of A, the fewer columns of them fit beside a piece of W
  if constexpr (MT <= 4)
    if (K > 1024) return launch_few_x<MT, 8, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
  if constexpr (MT <= 8)
    if (K > 512) return launch_few_x<MT, 16, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
  return launch_few_x<MT, 32, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
}

template <int VEC>
int launch_few_m(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K, int rows, int sms, int pdl, cudaStream_t st) {
  if (M == 1) return launch_few_r<1, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
  if (M == 2) return launch_few_r<2, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
  if (M <= 4) return launch_few_r<4, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
  if (rows == 8) return launch_few_r<8, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
  return launch_few_r<16, VEC>(A, lda, W, C, ldc, M, N, K, sms, pdl, st);
}

// ---------------------------------------------------------------------------- many rows
// Bound by the operands' way out of shared memory (128 bytes a clock: a thread's 8 x 4 sums read 12 floats for 32
// multiply-adds, 47 TFLOP/s at most; 41 to 44 measured).  128 threads compute 64 x 64 outputs, 8 x 4 each.  Slices of
// 16 k lie k-major in two buffers, so that a thread's rows and columns are 16-byte words; the operands of the next k are
// read while this one multiplies.  A thread copies the words that it will turn over itself three slices ahead into a
// ring of its own (no barrier): 0.64 us a slice where one slice ahead in registers took 1.05.  128 x 64 outputs, 8 x 8 a
// thread, measured slower at every size but one (2,048 x 32,768 over 1,024: 3.31 ms against 3.19): two blocks an SM.
constexpr int BM = 64, BN = 64, BK = 16, TM = 8, TN = 4, TILE_THREADS = 128, RING = 4;
constexpr int RING_BYTES = RING * (BM + BN) * BK * 4;

template <int VEC>
__global__ void __launch_bounds__(TILE_THREADS) gemm_f32_tile_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W,
                                                                  float* __restrict__ C, int ldc, int M, int N, int K) {
  constexpr int TX = BN / TN, PA = BM * BK / TILE_THREADS, PW = BN * BK / TILE_THREADS;
  static_assert(TX * (BM / TM) == TILE_THREADS, "a thread for every 8 x TN outputs");
  extern __shared__ float4 smem4[];
  __shared__ __align__(16) float As[2][BK][BM + 4];
  __shared__ __align__(16) float Ws[2][BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid % TX, ty = tid / TX;      // rows 4 ty + i and 32 + 4 ty + i, columns 4 tx + j
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  float* const ring = reinterpret_cast<float*>(smem4) + tid * 4;      // [RING][(PA + PW) / 4][threads] of 4 floats
  const int slices = (K + BK - 1) / BK, per_chunk = K <= ONE_CHAIN ? slices : CH / BK;
  int to_go = per_chunk;
  auto fetch4 = [&](float* to, const float* base, int ld, int row, int rows, int k) {
    const float* p = base + (size_t)row * ld + k;
#pragma unroll
    for (int j = 0; j < 4; j += VEC) copy_async<VEC>(to + j, row < rows && k + j < K ? p + j : base, row < rows && k + j < K);
  };
  auto fetch = [&](int s) {
    if (s < slices) {
      float* to = ring + (s % RING) * (PA + PW) * TILE_THREADS;
      const int k = s * BK + (tid % 4) * 4;
#pragma unroll
      for (int i = 0; i < PA / 4; ++i, to += 4 * TILE_THREADS) fetch4(to, A, lda, m0 + tid / 4 + i * (TILE_THREADS / 4), M, k);
#pragma unroll
      for (int i = 0; i < PW / 4; ++i, to += 4 * TILE_THREADS) fetch4(to, W, K, n0 + tid / 4 + i * (TILE_THREADS / 4), N, k);
    }
    copies_commit();
  };
  auto put = [&](int s) {
    const float* from = ring + (s % RING) * (PA + PW) * TILE_THREADS;
#pragma unroll
    for (int i = 0; i < (PA + PW) / 4; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(from + i * 4 * TILE_THREADS);
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (i < PA / 4) As[s & 1][(tid % 4) * 4 + j][tid / 4 + i * (TILE_THREADS / 4)] = f[j];
        else Ws[s & 1][(tid % 4) * 4 + j][tid / 4 + (i - PA / 4) * (TILE_THREADS / 4)] = f[j];
      }
    }
  };
  float a[2][TM], w[2][TN];
  auto operands = [&](int to, int b, int kk) {
    *reinterpret_cast<float4*>(a[to]) = *reinterpret_cast<const float4*>(&As[b][kk][ty * 4]);
    *reinterpret_cast<float4*>(a[to] + 4) = *reinterpret_cast<const float4*>(&As[b][kk][BM / 2 + ty * 4]);
    *reinterpret_cast<float4*>(w[to]) = *reinterpret_cast<const float4*>(&Ws[b][kk][tx * 4]);
  };
  float total[TM][TN], acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) total[i][j] = acc[i][j] = 0.f;
  static_assert(RING == 4, "three slices on their way");
  fetch(0);
  fetch(1);
  fetch(2);
  copies_wait<2>();
  put(0);
  __syncthreads();
  operands(0, 0, 0);
  for (int s = 0; s < slices; ++s) {
    const int b = s & 1;
    const bool more = s + 1 < slices;
    fetch(s + 3);              // into the words that this thread turned over before
    copies_wait<2>();          // its words of slice s + 1 are here
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      if (kk + 1 < BK) {
        operands((kk + 1) & 1, b, kk + 1);
      } else if (more) {
        put(s + 1);            // every thread left that buffer before the barrier behind it
        __syncthreads();
        operands(0, b ^ 1, 0);
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[kk & 1][i], w[kk & 1][j], acc[i][j]);
    }
    if (--to_go == 0 || !more) {   // the chunk is complete
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) { total[i][j] += acc[i][j]; acc[i][j] = 0.f; }
      to_go = per_chunk;
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i / 4) * (BM / 2) + ty * 4 + i % 4;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * ldc + n] = total[i][j];
    }
  }
}

template <int VEC>
int launch_tile(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K, cudaStream_t st) {
  const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) return DRYFT_ERR_UNSUPPORTED;
  const auto kern = gemm_f32_tile_kernel<VEC>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES);
  if (e != cudaSuccess) return (int)e;
  kern<<<grid, TILE_THREADS, RING_BYTES, st>>>(A, lda, W, C, ldc, M, N, K);
  return launch_status();
}

// Rows a block of the kernel for few rows, 0 for the tiles.  N = K = 1,024: one wave of blocks of 8 rows takes 5.6 us (up
// to 16 rows), of 16 rows 11.6 (up to 64 rows; 22 in two waves at 128), the tiles 42 from one row to 432.  N = 4,096: 22.6,
// 32.8 and 43 us at 24, 48 and 64 rows (two, three and four waves) against 42.  So the tiles start behind three waves; up
// to 16 rows the kernel for few is the faster one whatever N (a vocabulary of 32,768: 64 us against 121).
int few_rows(int M, int N, int K, int sms) {
  auto blocks = [&](int rows, int r) { return (long long)((M + rows - 1) / rows) * ((N + r - 1) / r); };
  if (M <= 8 || blocks(8, K > 512 ? 16 : 32) <= sms) return 8;
  return M <= 16 || blocks(16, 32) <= 3LL * sms ? 16 : 0;
}
}  // namespace

DRYFT_API int dryft_gemm_nt_f32(const float* A, int lda, const float* W, float* C, int ldc, int M, int N, int K,
                                int pdl, cudaStream_t st) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return DRYFT_ERR_UNSUPPORTED;
  // 16-byte accesses where every row of both operands starts on one
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int rows = K <= ONE_CHAIN ? 0 : few_rows(M, N, K, sms);
  if (rows)
    return vec ? launch_few_m<4>(A, lda, W, C, ldc, M, N, K, rows, sms, pdl, st)
               : launch_few_m<1>(A, lda, W, C, ldc, M, N, K, rows, sms, pdl, st);
  return vec ? launch_tile<4>(A, lda, W, C, ldc, M, N, K, st) : launch_tile<1>(A, lda, W, C, ldc, M, N, K, st);
}
