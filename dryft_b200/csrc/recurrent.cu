// Mixers whose memory is a fixed-size 32-bit state per sequence instead of cached keys: a step runs the tokens it is
// given from the state the step before left, and leaves the state for the next (one token, a prompt, or a piece of one).
//
// retention_scan     linear attention with one fixed decay per head, no softmax and no denominator.  Per head, with the
//                    rotated query q_t, the rotated key k_t times k_scale, and the value v_t of token t:
//                        S_t = decay * S_(t-1) + k_t v_t^T          S [dim, vdim], 32-bit
//                        o_t = S_t^T q_t ;  o_t <- o_t / sqrt(mean(o_t^2) + eps) ;  out = T( o_t * silu(g_t) )
//                    One block per (sequence, head) walks the sequence's tokens in order with S in shared memory.
//                    q | k | v | g are columns of one projection row (offsets given); the rotation pairs entry i with
//                    entry i + R/2 of the first R entries (angle = position * inv_freq[i]; see sincos_split below).
//
// rglru_gates        the input side of a real-gated linear recurrent unit over C channels in `blocks` equal groups:
//                        x_t  = xproj_t + x_bias                                   (a column range of the projection row)
//                        u_t  = conv_b + sum_j conv_w[c][j] * x_(t - (taps-1) + j)    (causal, per channel; inputs before
//                               the step come from the sequence's stored tail, zeros before the sequence's start)
//                        r_t  = sigmoid(Wa[b] u_t,b + ba) ;  i_t = sigmoid(Wi[b] u_t,b + bi)     (per group b, 32-bit)
//                        log a_t = -c * r_t * softplus(lam) ;  a_t = exp(log a_t)
//                        b_t  = sqrt(1 - a_t^2) * i_t * u_t          (1 - a^2 as -expm1(2 log a): no cancellation)
//                    leaves e_t = a_t - 1 (as expm1(log a_t): a decay of 0.9999 keeps its distance from one, which a
//                    32-bit a_t would round to one part in 2,000) and b_t, [tokens, C] in 32-bit.
// rglru_scan         S_t = S_(t-1) + (e_t * S_(t-1) + b_t) per channel, out_t = T( S_t * gelu_tanh(yproj_t + y_bias) ), then the new
//                    state and the new tail (the last taps-1 inputs) are stored.  Time is walked by eight warps at once,
//                    each folding its own steps first (see the kernel).
//
// Everything that enters a recurrence is 32-bit whatever the activation type T.  Sizes are runtime arguments of any value
// (shared memory permitting).  No block waits on another.
#include "common.cuh"
#include <math.h>

namespace {
constexpr int RT_THREADS = 256;

// a value that a launch before this one wrote (see common.cuh)
__device__ __forceinline__ float prev(const float* p) { return ld_prev(p); }
__device__ __forceinline__ float prev(const __nv_bfloat16* p) { return ld_prev_bf16(p); }

// sin and cos of  pos * (f_hi + f_lo)  for a rotary position: the product is formed in 32-bit, and what its rounding
// drops (recovered exactly with one fused multiply-add) plus the low half of the frequency are applied as a first-order
// turn, so the angle is as good as the frequency pair instead of losing one part in 2^24 of a large angle.  f_lo = 0 gives
// the plain 32-bit angle to within that correction.
__device__ __forceinline__ void sincos_split(float pos, float f_hi, float f_lo, float* sn, float* cs) {
  const float a = pos * f_hi;
  const float e = fmaf(pos, f_hi, -a) + pos * f_lo;
  float s, c;
  sincosf(a, &s, &c);
  *sn = fmaf(e, c, s);
  *cs = fmaf(-e, s, c);
}


template <typename T>
__global__ void __launch_bounds__(RT_THREADS) retention_scan_kernel(
    const T* __restrict__ proj, int ld, int q_off, int k_off, int v_off, int g_off, const int* __restrict__ cu_q,
    const int* __restrict__ seq_slot, const int* __restrict__ tok_pos, const float* __restrict__ inv_freq,
    const float* __restrict__ inv_freq_lo, int rot, const double* __restrict__ decay, float* __restrict__ state,
    T* __restrict__ out, int H, int dim, int vdim, float k_scale, float eps) {
  let_next_launch_in();   // a product behind this launch may start on its weights
  extern __shared__ __align__(16) float smem[];
  const int b = blockIdx.x, hd = blockIdx.y;
  const int slot = seq_slot[b];
  if (slot < 0) return;
  const int n0 = cu_q[b], n1 = cu_q[b + 1];
  const int cols = vdim < RT_THREADS ? vdim : RT_THREADS;   // threads side by side over the value index
  const int groups = RT_THREADS / cols;                      // groups of them over the key index
  float* S = smem;                        // [dim][vdim]
  float* qs = S + (size_t)dim * vdim;     // [dim]
  float* ks = qs + dim;                   // [dim]
  float* vs = ks + dim;                   // [vdim]
  float* red = vs + vdim;                 // [groups][vdim]
  __shared__ float scratch[33];
  const int tid = threadIdx.x;
  float* Sg = state + ((size_t)slot * H + hd) * dim * vdim;
  for (int i = tid; i < dim * vdim; i += RT_THREADS) S[i] = Sg[i];
  // the decay as a 32-bit value and what that drops: compounded over hundreds of tokens, one part in 2^24 of it shows
  const float dec = (float)decay[hd], dec_lo = (float)(decay[hd] - (double)dec);
  const int half = rot >> 1;
  const int cv = tid % cols, rg = tid / cols;
  const bool active = rg < groups;
  for (int n = n0; n < n1; ++n) {
    const T* row = proj + (size_t)n * ld;
    const float pos = (float)tok_pos[n];
    __syncthreads();   // the token before is done with qs / ks / vs / red
    for (int i = tid; i < 2 * dim; i += RT_THREADS) {
      const bool is_k = i >= dim;
      const int d = is_k ? i - dim : i;
      const T* src = row + (is_k ? k_off : q_off) + hd * dim;
      float val = to_f32<T>(src[d]);
      if (d < rot) {
        const int j = d < half ? d : d - half;
        const float other = to_f32<T>(src[d < half ? d + half : d - half]);
        float sn, cs;
        sincos_split(pos, inv_freq[j], inv_freq_lo ? inv_freq_lo[j] : 0.f, &sn, &cs);
        val = d < half ? val * cs - other * sn : val * cs + other * sn;
      }
      if (is_k) ks[d] = val * k_scale; else qs[d] = val;
    }
    for (int i = tid; i < vdim; i += RT_THREADS) vs[i] = to_f32<T>(row[v_off + hd * vdim + i]);
    __syncthreads();
    if (active) {
      for (int v = cv; v < vdim; v += cols) {
        const float vv = vs[v];
        float acc = 0.f;
        for (int d = rg; d < dim; d += groups) {
          const float old = S[d * vdim + v];
          const float s = fmaf(dec, old, fmaf(dec_lo, old, ks[d] * vv));
          S[d * vdim + v] = s;
          acc = fmaf(s, qs[d], acc);
        }
        red[rg * vdim + v] = acc;
      }
    }
    __syncthreads();
    float ss = 0.f;
    for (int v = tid; v < vdim; v += RT_THREADS) {
      float o = 0.f;
      for (int g = 0; g < groups; ++g) o += red[g * vdim + v];
      vs[v] = o;          // vs is free again: every thread passed the barrier above
      ss = fmaf(o, o, ss);
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.f / sqrtf(ss / (float)vdim + eps);
    for (int v = tid; v < vdim; v += RT_THREADS) {
      const float g = to_f32<T>(row[g_off + hd * vdim + v]);
      out[(size_t)n * H * vdim + hd * vdim + v] = from_f32<T>(vs[v] * inv * (g / (1.f + expf(-g))));
    }
  }
  __syncthreads();
  for (int i = tid; i < dim * vdim; i += RT_THREADS) Sg[i] = S[i];
}

// The same for steps in which every sequence brings one token (token b is sequence b's): bound by one trip to memory for a head's state.
// A thread holds up to STEP_ROWS rows' 16-byte words of it in registers, all requested at once, and works the angles out meanwhile; rows are
// summed in order by each thread, threads in order.  `early`: the words are requested before the launch before this one is waited for.  That
// is right only where whatever wrote the state last was complete before this step's first overlapped launch: a run step's own state, which
// the step before wrote.  A state that an earlier run step of the same step wrote (or two direct calls in a row) is read behind the wait:
// every launch in between may have signalled at its start, and then nothing else orders that write before this read.
// 16 heads of 128 x 128, one token: 11.1 us a launch with the walk above, 9.7 here, of which half runs beside the product before it (5.2 us of
// its own): a 1,300-token prompt + 16 steps, 6 such launches a step, 14,709 -> 14,266 us.  Sizes it does not take (rows that are no 16-byte words, more
// than STEP_ROWS rows a thread, angles or partial sums beyond 48 KB of shared memory) are walked as longer steps are.
// Few rows a thread have a kernel with registers for as many: 64 sequences, us with registers for 16 rows / now / the walk: 8 heads of
// 64 x 64 (four rows a thread) 9.1 / 5.7 / 7.6, 32 heads of 16 x 32 (one) 25.8 / 11.4 / 12.3, 16 heads of 64 x 128 (eight) 25.2 / 18.0 / 23.4.
constexpr int STEP_ROWS = 16;
__host__ __device__ constexpr int step_rows(int dim, int vdim) { return (dim + RT_THREADS / (vdim / 4) - 1) / (RT_THREADS / (vdim / 4)); }
__host__ __device__ constexpr bool step_fits(int dim, int vdim, int rot) {
  return vdim % 4 == 0 && vdim <= 4 * RT_THREADS && step_rows(dim, vdim) <= STEP_ROWS && rot <= 1024;
}

template <typename T, int ROWS>
__global__ void __launch_bounds__(RT_THREADS) retention_step_kernel(
    const T* __restrict__ proj, int ld, int q_off, int k_off, int v_off, int g_off, const int* __restrict__ seq_slot, const int* __restrict__ tok_pos,
    const float* __restrict__ inv_freq, const float* __restrict__ inv_freq_lo, int rot, const double* __restrict__ decay, float* __restrict__ state,
    T* __restrict__ out, int H, int dim, int vdim, float k_scale, float eps, int early) {
  let_next_launch_in();   // a product behind this launch may start on its weights
  extern __shared__ __align__(16) float smem[];
  const int b = blockIdx.x, hd = blockIdx.y, tid = threadIdx.x;
  const int slot = seq_slot[b];
  if (slot < 0) {      // (waits too: a launch of padding alone must not be complete before the launch before it)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  const int words = vdim / 4, groups = RT_THREADS / words, cv = tid % words, rg = tid / words, half = rot >> 1;
  float4* const red = reinterpret_cast<float4*>(smem);      // [groups][words]
  float* const qs = smem + (size_t)groups * vdim;           // [dim]
  float* const ks = qs + dim;                               // [dim]
  float* const vs = smem + ((size_t)groups * vdim + 2 * dim + 3) / 4 * 4;      // [vdim]
  float2* const turn = reinterpret_cast<float2*>(vs + vdim);      // [rot / 2] sin, cos
  __shared__ float scratch[33];
  float4* const Sg = reinterpret_cast<float4*>(state + ((size_t)slot * H + hd) * dim * vdim);
  float4 old[ROWS];
  auto request = [&]() {      // (through L2: a state written while this launch was resident is no read-only data)
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int d = rg + i * groups;
      old[i] = rg < groups && d < dim ? __ldcg(Sg + (size_t)d * words + cv) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  if (early) request();
  // the decay as a 32-bit value and what that drops, as above
  const float dec = (float)decay[hd], dec_lo = (float)(decay[hd] - (double)dec);
  const float pos = (float)tok_pos[b];
#pragma unroll 1
  for (int j = tid; j < half; j += RT_THREADS) {
    float sn, cs;
    sincos_split(pos, inv_freq[j], inv_freq_lo ? inv_freq_lo[j] : 0.f, &sn, &cs);
    turn[j] = make_float2(sn, cs);
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");      // the projection; what it wrote is read through L2
  if (!early) request();
  const T* const row = proj + (size_t)b * ld;
#pragma unroll 1
  for (int i = tid; i < 2 * dim; i += RT_THREADS) {
    const bool is_k = i >= dim;
    const int d = is_k ? i - dim : i, partner = d < half ? d + half : d - half;
    const T* const src = row + (is_k ? k_off : q_off) + hd * dim;
    float val = prev(src + d);
    if (d < rot) {
      const float2 t = turn[d < half ? d : d - half];
      const float other = prev(src + partner);
      val = d < half ? val * t.y - other * t.x : val * t.y + other * t.x;
    }
    if (is_k) ks[d] = val * k_scale; else qs[d] = val;
  }
#pragma unroll 1
  for (int i = tid; i < vdim; i += RT_THREADS) vs[i] = prev(row + v_off + hd * vdim + i);
  float gate = tid < vdim ? prev(row + g_off + hd * vdim + tid) : 0.f;
  __syncthreads();
  if (rg < groups) {
    const float4 v = reinterpret_cast<const float4*>(vs)[cv];
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int d = rg + i * groups;
      if (d < dim) {
        const float k = ks[d], q = qs[d];
        float4 n;
        n.x = fmaf(dec, old[i].x, fmaf(dec_lo, old[i].x, k * v.x));
        n.y = fmaf(dec, old[i].y, fmaf(dec_lo, old[i].y, k * v.y));
        n.z = fmaf(dec, old[i].z, fmaf(dec_lo, old[i].z, k * v.z));
        n.w = fmaf(dec, old[i].w, fmaf(dec_lo, old[i].w, k * v.w));
        Sg[(size_t)d * words + cv] = n;
        acc.x = fmaf(n.x, q, acc.x);
        acc.y = fmaf(n.y, q, acc.y);
        acc.z = fmaf(n.z, q, acc.z);
        acc.w = fmaf(n.w, q, acc.w);
      }
    }
    red[rg * words + cv] = acc;
  }
  __syncthreads();
  float ss = 0.f;
#pragma unroll 1
  for (int v = tid; v < vdim; v += RT_THREADS) {
    float o = 0.f;
#pragma unroll 4
    for (int g = 0; g < groups; ++g) o += smem[(size_t)g * vdim + v];
    vs[v] = o;          // vs is free again: every thread passed the barrier above
    ss = fmaf(o, o, ss);
  }
  ss = block_sum(ss, scratch);
  const float inv = 1.f / sqrtf(ss / (float)vdim + eps);
#pragma unroll 1
  for (int v = tid; v < vdim; v += RT_THREADS) {
    if (v != tid) gate = prev(row + g_off + hd * vdim + v);
    out[(size_t)b * H * vdim + hd * vdim + v] = from_f32<T>(vs[v] * inv * (gate / (1.f + expf(-gate))));
  }
}

// ---------------------------------------------------------------------------------------------------------------------
// The same retention for steps of many tokens, in chunks of CH tokens so that the work is matrix-shaped and spread over
// (chunk, head) blocks instead of walked token by token.  For chunk g of a sequence, L tokens long, with S_in the state
// before it (w = decay):
//     D_g   = sum_j w^(L-1-j) k_j v_j^T                                   retention_chunk_state   (every chunk at once)
//     S_in  of every chunk, by S <- w^L S + D_g in order                   retention_chunk_prefix  (elementwise; the
//                                                                          sequence's stored state is read and updated)
//     o_i   = w^(i+1) S_in^T q_i + sum_(j<=i) w^(i-j) (q_i . k_j) v_j       retention_chunk_out     (every chunk at once),
// then the same norm and gate as above.  Powers of the decay come from a table made in 64-bit.  Chunk g of the step is
// found from cu_q: sequence b has ceil(len_b / CH) chunks, numbered in sequence order after those of the sequences before.
constexpr int CH = 64;
constexpr int CK_THREADS = 256;

__device__ __forceinline__ bool locate_chunk(const int* __restrict__ cu_q, int n_seqs, int g, int* b_out, int* k_out) {
  int base = 0;
  for (int b = 0; b < n_seqs; ++b) {
    const int nc = (cu_q[b + 1] - cu_q[b] + CH - 1) / CH;
    if (g < base + nc) { *b_out = b; *k_out = g - base; return true; }
    base += nc;
  }
  return false;
}

// (sin, cos) of every token's angles, [n_tokens][rot / 2]: worked out once a launch of the chunked form.  Every head's blocks
// of both products evaluated them anew before, which was a third of those blocks' time.
__global__ void retention_angles_kernel(const int* __restrict__ tok_pos, const float* __restrict__ inv_freq, const float* __restrict__ inv_freq_lo,
                                        float2* __restrict__ angles, int n_tokens, int half) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_tokens * half) return;
  const int n = i / half, j = i - n * half;
  float sn, cs;
  sincos_split((float)tok_pos[n], inv_freq[j], inv_freq_lo ? inv_freq_lo[j] : 0.f, &sn, &cs);
  angles[i] = make_float2(sn, cs);
}

// rows [L][ld] of shared memory <- the rotated (and scaled) head vectors of L tokens; columns dim..ld-1 are zeroed.  A warp a row, a
// lane both halves of a rotated pair.  `last_first`: a row's further factor, last_first[L - 1 - t].
template <typename T>
__device__ __forceinline__ void load_rotated(float* dst, int ld, const T* __restrict__ proj, int ldp, int col0, int n_first, int L,
                                             int dim, int rot, const float2* __restrict__ angles, float scale, const float* last_first = nullptr) {
  const int half = rot >> 1, lane = threadIdx.x & 31;
  for (int t = threadIdx.x >> 5; t < L; t += CK_THREADS / 32) {
    const T* src = proj + (size_t)(n_first + t) * ldp + col0;
    const float2* ang = angles + (size_t)(n_first + t) * half;
    float* to = dst + t * ld;
    const float more = last_first ? last_first[L - 1 - t] : 1.f;
#pragma unroll 2
    for (int d = lane; d < half; d += 32) {
      const float a = to_f32<T>(src[d]), b = to_f32<T>(src[d + half]);
      const float2 sc = ang[d];
      float u = (a * sc.y - b * sc.x) * scale, v = (b * sc.y + a * sc.x) * scale;
      if (last_first) { u *= more; v *= more; }
      to[d] = u;
      to[d + half] = v;
    }
    for (int d = rot + lane; d < ld; d += 32) {
      float u = d < dim ? to_f32<T>(src[d]) * scale : 0.f;
      if (last_first) u *= more;
      to[d] = u;
    }
  }
}
template <typename T>
__device__ __forceinline__ void load_values(float* dst, int ld, const T* __restrict__ proj, int ldp, int col0, int n_first, int L, int rows, int vdim) {
  const int lane = threadIdx.x & 31;
  for (int t = threadIdx.x >> 5; t < rows; t += CK_THREADS / 32) {
    const T* src = proj + (size_t)(n_first + t) * ldp + col0;
#pragma unroll 4
    for (int v = lane; v < ld; v += 32) dst[t * ld + v] = t < L && v < vdim ? to_f32<T>(src[v]) : 0.f;
  }
}

template <typename T>
__global__ void __launch_bounds__(CK_THREADS) retention_chunk_state_kernel(
    const T* __restrict__ proj, int ld, int k_off, int v_off, const int* __restrict__ cu_q, const int* __restrict__ seq_slot,
    int n_seqs, const float2* __restrict__ angles, int rot, const double* __restrict__ decay, float* __restrict__ sbuf, int H, int dim,
    int vdim, float k_scale) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int loc[3];
  const int g = blockIdx.x, hd = blockIdx.y;
  if (threadIdx.x == 0) {
    int b = 0, k = 0;
    loc[2] = locate_chunk(cu_q, n_seqs, g, &b, &k) && seq_slot[b] >= 0;
    loc[0] = b; loc[1] = k;
  }
  __syncthreads();
  if (!loc[2]) return;
  const int b = loc[0], n_first = cu_q[b] + loc[1] * CH, L = min(CH, cu_q[b + 1] - n_first);
  const int dP = (dim + 7) & ~7, vP = (vdim + 7) & ~7;
  float* ks = smem;                 // [CH][dP]
  float* vs = ks + CH * dP;         // [CH][vP]
  float* pw = vs + CH * vP;         // [CH + 1]
  for (int i = threadIdx.x; i <= CH; i += CK_THREADS) pw[i] = (float)pow(decay[hd], (double)i);
  __syncthreads();
  load_rotated<T>(ks, dP, proj, ld, k_off + hd * dim, n_first, L, dim, rot, angles, k_scale, pw);
  load_values<T>(vs, vP, proj, ld, v_off + hd * vdim, n_first, L, L, vdim);
  __syncthreads();
  float* dst = sbuf + ((size_t)g * H + hd) * dim * vdim;
  const int tv = vP / 8, n_tiles = (dP / 8) * tv;
  for (int tile = threadIdx.x; tile < n_tiles; tile += CK_THREADS) {
    const int d0 = (tile / tv) * 8, v0 = (tile % tv) * 8;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[i][c] = 0.f;
#pragma unroll 4
    for (int j = 0; j < L; ++j) {
      const float4 k0 = *reinterpret_cast<const float4*>(ks + j * dP + d0), k1 = *reinterpret_cast<const float4*>(ks + j * dP + d0 + 4);
      const float4 u0 = *reinterpret_cast<const float4*>(vs + j * vP + v0), u1 = *reinterpret_cast<const float4*>(vs + j * vP + v0 + 4);
      const float kv[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w}, vv[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[i][c] = fmaf(kv[i], vv[c], acc[i][c]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c < 8; ++c)
        if (d0 + i < dim && v0 + c < vdim) dst[(size_t)(d0 + i) * vdim + v0 + c] = acc[i][c];
  }
}

__global__ void retention_chunk_prefix_kernel(const int* __restrict__ cu_q, const int* __restrict__ seq_slot,
                                              const double* __restrict__ decay, float* __restrict__ sbuf,
                                              float* __restrict__ state, int H, int per_head) {
  const int b = blockIdx.x, hd = blockIdx.y;
  const int e = blockIdx.z * blockDim.x + threadIdx.x;
  const int slot = seq_slot[b];
  if (slot < 0 || e >= per_head) return;
  int base = 0;
  for (int bb = 0; bb < b; ++bb) base += (cu_q[bb + 1] - cu_q[bb] + CH - 1) / CH;
  const int q = cu_q[b + 1] - cu_q[b];
  float* sp = state + ((size_t)slot * H + hd) * per_head + e;
  float S = *sp;
  const double w = decay[hd];
  const float w_full = (float)pow(w, (double)CH);
  const int n_chunks = (q + CH - 1) / CH;
  for (int k0 = 0; k0 < n_chunks; k0 += 8) {   // eight chunk sums asked for at once, then folded in order
    float delta[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (k0 + u < n_chunks) delta[u] = __ldcs(sbuf + ((size_t)(base + k0 + u) * H + hd) * per_head + e);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if (k0 + u < n_chunks) {
        sbuf[((size_t)(base + k0 + u) * H + hd) * per_head + e] = S;   // the state the chunk starts from
        const int L = min(CH, q - (k0 + u) * CH);
        S = fmaf(L == CH ? w_full : (float)pow(w, (double)L), S, delta[u]);
      }
    }
  }
  *sp = S;
}

template <typename T>
__global__ void __launch_bounds__(CK_THREADS) retention_chunk_out_kernel(
    const T* __restrict__ proj, int ld, int q_off, int k_off, int v_off, int g_off, const int* __restrict__ cu_q,
    const int* __restrict__ seq_slot, int n_seqs, const float2* __restrict__ angles, int rot, const double* __restrict__ decay,
    const float* __restrict__ sbuf, T* __restrict__ out, int H, int dim, int vdim, float k_scale, float eps) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int loc[3];
  const int g = blockIdx.x, hd = blockIdx.y;
  if (threadIdx.x == 0) {
    int b = 0, k = 0;
    loc[2] = locate_chunk(cu_q, n_seqs, g, &b, &k) && seq_slot[b] >= 0;
    loc[0] = b; loc[1] = k;
  }
  __syncthreads();
  if (!loc[2]) return;
  const int b = loc[0], n_first = cu_q[b] + loc[1] * CH, L = min(CH, cu_q[b + 1] - n_first);
  const int dQ = ((dim + 3) & ~3) + 1;           // odd row length: rows of q and k fall on different banks
  const int vP = (vdim + 3) & ~3;
  const int stage = max(CH * dQ, CH * vP);       // the q rows' place also holds the outputs before the norm
  float* vs = smem;                  // [CH][vP]            (16-byte rows first)
  float* slab = vs + CH * vP;        // [SLAB][vP]          a slab of the state the chunk starts from
  float* qs = slab + 16 * vP;        // [CH][dQ], later o [CH][vP]
  float* ks = qs + stage;            // [CH][dQ]
  float* A = ks + CH * dQ;           // [CH][CH + 1]
  float* pw = A + CH * (CH + 1);     // [CH + 1]
  for (int i = threadIdx.x; i <= CH; i += CK_THREADS) pw[i] = (float)pow(decay[hd], (double)i);
  load_rotated<T>(qs, dQ, proj, ld, q_off + hd * dim, n_first, L, dim, rot, angles, 1.f);
  load_rotated<T>(ks, dQ, proj, ld, k_off + hd * dim, n_first, L, dim, rot, angles, k_scale);
  load_values<T>(vs, vP, proj, ld, v_off + hd * vdim, n_first, L, CH, vdim);
  for (int idx = threadIdx.x + L * dQ; idx < CH * dQ; idx += CK_THREADS) { qs[idx] = 0.f; ks[idx] = 0.f; }   // rows behind the chunk
  __syncthreads();
  // A[i][j] = w^(i-j) q_i . k_j  for j <= i, else 0: 4 x 4 outputs a thread
  for (int tile = threadIdx.x; tile < (CH / 4) * (CH / 4); tile += CK_THREADS) {
    const int i0 = (tile / (CH / 4)) * 4, j0 = (tile % (CH / 4)) * 4;
    float acc[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
    if (j0 <= i0 + 3 && i0 < L) {
#pragma unroll 4
      for (int d = 0; d < dim; ++d) {
        float qv[4], kv[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) { qv[r] = qs[(i0 + r) * dQ + d]; kv[r] = ks[(j0 + r) * dQ + d]; }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[r][c] = fmaf(qv[r], kv[c], acc[r][c]);
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int i = i0 + r, j = j0 + c;
        A[i * (CH + 1) + j] = j <= i ? acc[r][c] * pw[i - j] : 0.f;
      }
  }
  __syncthreads();
  // o = w^(i+1) (q S_in) + A v : 8 rows x 4 columns a thread, kept in registers until every thread has read q.
  // S_in comes through shared memory in slabs of SLAB key rows; the next slab is asked for (into registers) before the
  // current one is multiplied, so its trip from L2 hides behind the products.
  const float* S_in = sbuf + ((size_t)g * H + hd) * dim * vdim;
  const int tv = vP / 4, n_tiles = (CH / 8) * tv;
  constexpr int MAX_TILES = 4;       // tiles a thread may hold (value sizes up to 512)
  constexpr int SLAB = 16, SLAB_LOADS = (SLAB * 512 / 4 + CK_THREADS - 1) / CK_THREADS;   // float4 pieces a thread fetches
  float acc[MAX_TILES][8][4];
#pragma unroll
  for (int t = 0; t < MAX_TILES; ++t)
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[t][r][c] = 0.f;
  const int slab_vec = SLAB * tv;    // float4 pieces of a slab [SLAB][vP]
  const bool rows_vec = (vdim & 3) == 0;
  float4 pre[SLAB_LOADS];
  auto fetch = [&](int d0) {
#pragma unroll
    for (int u = 0; u < SLAB_LOADS; ++u) {
      const int idx = threadIdx.x + u * CK_THREADS;
      pre[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (idx < slab_vec) {
        const int dd = d0 + idx / tv, v = (idx % tv) * 4;
        if (dd < dim) {
          const float* src = S_in + (size_t)dd * vdim + v;
          if (rows_vec) pre[u] = __ldg(reinterpret_cast<const float4*>(src));
          else pre[u] = make_float4(v < vdim ? __ldg(src) : 0.f, v + 1 < vdim ? __ldg(src + 1) : 0.f,
                                    v + 2 < vdim ? __ldg(src + 2) : 0.f, v + 3 < vdim ? __ldg(src + 3) : 0.f);
        }
      }
    }
  };
  fetch(0);
  for (int d0 = 0; d0 < dim; d0 += SLAB) {
    __syncthreads();   // the slab before is used up
#pragma unroll
    for (int u = 0; u < SLAB_LOADS; ++u) {
      const int idx = threadIdx.x + u * CK_THREADS;
      if (idx < slab_vec) *reinterpret_cast<float4*>(slab + (size_t)idx * 4) = pre[u];
    }
    __syncthreads();
    if (d0 + SLAB < dim) fetch(d0 + SLAB);
    const int d_end = min(SLAB, dim - d0);
    int n_mine = 0;
    for (int tile = threadIdx.x; tile < n_tiles && n_mine < MAX_TILES; tile += CK_THREADS, ++n_mine) {
      const int i0 = (tile / tv) * 8, v0 = (tile % tv) * 4;
      if (i0 >= L) continue;
      float (*a)[4] = acc[n_mine];
#pragma unroll 4
      for (int dd = 0; dd < d_end; ++dd) {
        const float4 sv = *reinterpret_cast<const float4*>(slab + (size_t)dd * vP + v0);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float qv = qs[(i0 + r) * dQ + d0 + dd];
          a[r][0] = fmaf(qv, sv.x, a[r][0]); a[r][1] = fmaf(qv, sv.y, a[r][1]);
          a[r][2] = fmaf(qv, sv.z, a[r][2]); a[r][3] = fmaf(qv, sv.w, a[r][3]);
        }
      }
    }
  }
  {
    int n_mine = 0;
    for (int tile = threadIdx.x; tile < n_tiles && n_mine < MAX_TILES; tile += CK_THREADS, ++n_mine) {
      const int i0 = (tile / tv) * 8, v0 = (tile % tv) * 4;
      if (i0 >= L) continue;
      float (*a)[4] = acc[n_mine];
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) a[r][c] *= pw[i0 + r + 1];
      const int j_end = min(L, i0 + 8);
#pragma unroll 4
      for (int j = 0; j < j_end; ++j) {
        const float4 vv = *reinterpret_cast<const float4*>(vs + (size_t)j * vP + v0);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float av = A[(i0 + r) * (CH + 1) + j];
          a[r][0] = fmaf(av, vv.x, a[r][0]); a[r][1] = fmaf(av, vv.y, a[r][1]);
          a[r][2] = fmaf(av, vv.z, a[r][2]); a[r][3] = fmaf(av, vv.w, a[r][3]);
        }
      }
    }
  }
  __syncthreads();   // q is read by all: its place takes the outputs
  int n_mine = 0;
  for (int tile = threadIdx.x; tile < n_tiles && n_mine < MAX_TILES; tile += CK_THREADS, ++n_mine) {
    const int i0 = (tile / tv) * 8, v0 = (tile % tv) * 4;
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) qs[(i0 + r) * vP + v0 + c] = acc[n_mine][r][c];
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int i = warp; i < L; i += CK_THREADS / 32) {
    float ss = 0.f;
    for (int v = lane; v < vdim; v += 32) { const float o = qs[i * vP + v]; ss = fmaf(o, o, ss); }
    ss = warp_sum(ss);
    const float inv = 1.f / sqrtf(ss / (float)vdim + eps);
    const size_t n = (size_t)(n_first + i);
    for (int v = lane; v < vdim; v += 32) {
      const float gv = to_f32<T>(proj[n * ld + g_off + hd * vdim + v]);
      out[n * H * vdim + hd * vdim + v] = from_f32<T>(qs[i * vP + v] * inv * (gv / (1.f + expf(-gv))));
    }
  }
}

constexpr int GT = 8;          // tokens a thread of rglru_gates adds up
constexpr int G_THREADS = 256;

// A block takes GT * groups tokens and one gate block: a thread an output of both gates for GT tokens, `groups` threads beside one
// another the same output for other tokens (two with gate blocks of 128, where half of the threads had nothing to do before).  The
// inputs lie token-fast in shared memory, two 16-byte broadcasts a k; eight k's weights are requested at a time.  AHEAD: the next
// eight while eight are used, for launches whose blocks all run at once with the registers that it takes (16 gate blocks of 128, 128
// tokens: 21 us without).
template <typename T, bool AHEAD>
__global__ void __launch_bounds__(G_THREADS) rglru_gates_kernel(
    const T* __restrict__ proj, int ld, int x_off, const float* __restrict__ x_bias, const int* __restrict__ tok_slot,
    const float* __restrict__ conv_w, const float* __restrict__ conv_b, int taps, const float* __restrict__ tail,
    const float* __restrict__ w_gates, const float* __restrict__ b_a, const float* __restrict__ b_i,
    const float* __restrict__ sp_lam, float c_mult, float* __restrict__ a_out, float* __restrict__ b_out, int n_tokens,
    int C, int nb, int groups) {
  extern __shared__ __align__(16) float u_s[];   // [groups][nb][GT]
  const int n0 = blockIdx.x * GT * groups, blk = blockIdx.y, c0 = blk * nb;
  const int K1 = taps - 1;
  for (int idx = threadIdx.x; idx < GT * groups * nb; idx += G_THREADS) {
    const int t = idx / nb, cc = idx - t * nb, n = n0 + t, c = c0 + cc;
    float u = 0.f;
    if (n < n_tokens) {
      const int slot = tok_slot[n];
      if (slot >= 0) {
        int avail = 0;   // tokens of the same sequence right before this one in the step, up to taps-1
        while (avail < K1 && n - avail - 1 >= 0 && tok_slot[n - avail - 1] == slot) ++avail;
        u = conv_b[c];
        for (int j = 0; j < taps; ++j) {
          const int back = K1 - j;
          float xv;
          if (back <= avail) xv = to_f32<T>(proj[(size_t)(n - back) * ld + x_off + c]) + x_bias[c];
          else xv = tail[((size_t)slot * K1 + (K1 - back + avail)) * C + c];
          u = fmaf(conv_w[(size_t)c * taps + j], xv, u);
        }
      }
    }
    u_s[((t / GT) * nb + cc) * GT + t % GT] = u;
  }
  __syncthreads();
  const float* wg = w_gates + (size_t)blk * nb * 2 * nb;   // [k][2][o]
  for (int i = threadIdx.x; i < nb * groups; i += G_THREADS) {
    const int g = i / nb, o = i - g * nb;
    const float* ug = u_s + (size_t)g * nb * GT;
    float ar[GT], ai[GT];
    const float ba = b_a[c0 + o], bi = b_i[c0 + o];
#pragma unroll
    for (int t = 0; t < GT; ++t) { ar[t] = ba; ai[t] = bi; }
    auto one = [&](int k, float wr, float wi) {
      const float4 u0 = *reinterpret_cast<const float4*>(ug + k * GT), u1 = *reinterpret_cast<const float4*>(ug + k * GT + 4);
      const float uv[GT] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
      for (int t = 0; t < GT; ++t) {
        ar[t] = fmaf(wr, uv[t], ar[t]);
        ai[t] = fmaf(wi, uv[t], ai[t]);
      }
    };
    int k = 0;
    if (AHEAD) {
      float wr[2][8], wi[2][8];
      auto request = [&](int to, int k0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) { wr[to][u] = wg[((size_t)(k0 + u) * 2) * nb + o]; wi[to][u] = wg[((size_t)(k0 + u) * 2 + 1) * nb + o]; }
      };
      if (nb >= 8) request(0, 0);
      for (; k + 8 <= nb; k += 8) {
        const int now = (k >> 3) & 1;
        if (now == 0) {
          if (k + 16 <= nb) request(1, k + 8);
#pragma unroll
          for (int u = 0; u < 8; ++u) one(k + u, wr[0][u], wi[0][u]);
        } else {
          if (k + 16 <= nb) request(0, k + 8);
#pragma unroll
          for (int u = 0; u < 8; ++u) one(k + u, wr[1][u], wi[1][u]);
        }
      }
    }
#pragma unroll 8
    for (; k < nb; ++k) one(k, wg[((size_t)k * 2) * nb + o], wg[((size_t)k * 2 + 1) * nb + o]);
    const float sp = sp_lam[c0 + o];
#pragma unroll
    for (int t = 0; t < GT; ++t) {
      const int n = n0 + g * GT + t;
      if (n >= n_tokens) break;
      const float r = 1.f / (1.f + expf(-ar[t])), ig = 1.f / (1.f + expf(-ai[t]));
      const float log_a = -c_mult * r * sp;
      a_out[(size_t)n * C + c0 + o] = expm1f(log_a);   // a - 1: a decay close to one keeps its distance from one
      b_out[(size_t)n * C + c0 + o] = sqrtf(-expm1f(2.f * log_a)) * ig * ug[o * GT + t];
    }
  }
}

__device__ __forceinline__ float gelu_tanh_f(float z) {
  return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// The same for few tokens, with the same order of additions (one chain along k), so that a token's gates do not depend on its company.
// There a block per gate block leaves a thread 2 nb dependent trips long (22 us for one token of 16 blocks of 128 x 128).  Here a block
// takes FEW_COLS of its outputs for up to NT tokens: the weights of FEW_K inputs come in one trip into shared memory, and a thread walks
// them for one output, one gate and NT / 4 tokens.
constexpr int FEW_COLS = 32, FEW_K = 128;
constexpr size_t few_smem(int tokens, int nb) { return sizeof(float) * ((size_t)tokens * nb + FEW_K * 2 * FEW_COLS); }

template <typename T, int NT>
__global__ void __launch_bounds__(G_THREADS) rglru_gates_few_kernel(
    const T* __restrict__ proj, int ld, int x_off, const float* __restrict__ x_bias, const int* __restrict__ tok_slot,
    const float* __restrict__ conv_w, const float* __restrict__ conv_b, int taps, const float* __restrict__ tail,
    const float* __restrict__ w_gates, const float* __restrict__ b_a, const float* __restrict__ b_i,
    const float* __restrict__ sp_lam, float c_mult, float* __restrict__ a_out, float* __restrict__ b_out, int n_tokens,
    int C, int nb, int vec) {
  extern __shared__ __align__(16) float few_s[];
  float* const w_s = few_s;                            // [FEW_K][2][FEW_COLS]
  float* const u_s = few_s + FEW_K * 2 * FEW_COLS;     // [nb][NT]
  __shared__ float logits[NT][2][FEW_COLS];
  const int n0 = blockIdx.x * NT, blk = blockIdx.y, c0 = blk * nb, o0 = blockIdx.z * FEW_COLS;
  const int K1 = taps - 1, live = min(NT, n_tokens - n0), cols = min(FEW_COLS, nb - o0);
  const float* wg = w_gates + (size_t)blk * nb * 2 * nb + o0;   // [k][2][o]
  constexpr int PER = FEW_K * 2 * FEW_COLS / G_THREADS;         // floats of a piece that a thread brings
  float wv[PER];
  auto request = [&](int k0) {        // thread -> (input, gate) row r of the piece, four or one neighbouring columns
    if (vec) {
#pragma unroll
      for (int j = 0; j < PER; j += 4) {
        const int i = (threadIdx.x + (j / 4) * G_THREADS) * 4, r = i / FEW_COLS, c = i % FEW_COLS;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k0 + r / 2 < nb && c < cols) v = *reinterpret_cast<const float4*>(wg + (size_t)(2 * k0 + r) * nb + c);
        wv[j] = v.x; wv[j + 1] = v.y; wv[j + 2] = v.z; wv[j + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int i = threadIdx.x + j * G_THREADS, r = i / FEW_COLS, c = i % FEW_COLS;
        wv[j] = k0 + r / 2 < nb && c < cols ? wg[(size_t)(2 * k0 + r) * nb + c] : 0.f;
      }
    }
  };
  auto put = [&] {
    if (vec) {
#pragma unroll
      for (int j = 0; j < PER; j += 4)
        *reinterpret_cast<float4*>(w_s + (threadIdx.x + (j / 4) * G_THREADS) * 4) = make_float4(wv[j], wv[j + 1], wv[j + 2], wv[j + 3]);
    } else {
#pragma unroll
      for (int j = 0; j < PER; ++j) w_s[threadIdx.x + j * G_THREADS] = wv[j];
    }
  };
  request(0);
  for (int idx = threadIdx.x; idx < NT * nb; idx += G_THREADS) {
    const int t = idx / nb, cc = idx % nb, n = n0 + t, c = c0 + cc;
    float u = 0.f;
    const int slot = t < live ? tok_slot[n] : -1;
    if (slot >= 0) {
      int avail = 0;   // tokens of the same sequence right before this one in the step, up to taps-1
      while (avail < K1 && n - avail - 1 >= 0 && tok_slot[n - avail - 1] == slot) ++avail;
      u = conv_b[c];
      for (int j = 0; j < taps; ++j) {
        const int back = K1 - j;
        float xv;
        if (back <= avail) xv = to_f32<T>(proj[(size_t)(n - back) * ld + x_off + c]) + x_bias[c];
        else xv = tail[((size_t)slot * K1 + (K1 - back + avail)) * C + c];
        u = fmaf(conv_w[(size_t)c * taps + j], xv, u);
      }
    }
    u_s[cc * NT + t] = u;
  }
  // warp -> gate and tokens, lane -> output
  constexpr int TW = NT >= 4 ? NT / 4 : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gate = warp & 1, t0 = (warp >> 1) * TW;
  const bool works = t0 < NT;
  float acc[TW];
#pragma unroll
  for (int t = 0; t < TW; ++t) acc[t] = lane < cols ? (gate ? b_i : b_a)[c0 + o0 + lane] : 0.f;
  for (int k0 = 0; k0 < nb; k0 += FEW_K) {
    if (k0 > 0) {
      __syncthreads();      // the piece before is used up
      request(k0);
    }
    put();
    __syncthreads();
    if (works) {
      const int ks = min(FEW_K, nb - k0);
#pragma unroll 16
      for (int k = 0; k < ks; ++k) {
        const float w = w_s[(2 * k + gate) * FEW_COLS + lane];
#pragma unroll
        for (int t = 0; t < TW; ++t) acc[t] = fmaf(w, u_s[(k0 + k) * NT + t0 + t], acc[t]);
      }
    }
  }
  if (works) {
#pragma unroll
    for (int t = 0; t < TW; ++t) logits[t0 + t][gate][lane] = acc[t];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < live * FEW_COLS; i += G_THREADS) {
    const int t = i / FEW_COLS, oo = i % FEW_COLS, n = n0 + t, c = o0 + oo;
    if (c >= nb) continue;
    const float r = 1.f / (1.f + expf(-logits[t][0][oo])), ig = 1.f / (1.f + expf(-logits[t][1][oo]));
    const float log_a = -c_mult * r * sp_lam[c0 + c];
    a_out[(size_t)n * C + c0 + c] = expm1f(log_a);   // a - 1: a decay close to one keeps its distance from one
    b_out[(size_t)n * C + c0 + c] = sqrtf(-expm1f(2.f * log_a)) * ig * u_s[c * NT + t];
  }
}
// The form for few tokens up to this many blocks a multiprocessor.  Against the other, 8 / 16 gate blocks of 128: 16.4 / 14.9 us and 21 /
// 19 at 512 blocks, 20 / 20 and 22 / 21 at 768, 26 / 26 and 23 / 22 at 1,024; 4 of 256: 29 and 37, 37 and 37, 47 and 37.
constexpr int FEW_BLOCKS_PER_SM = 5;

// A block takes 32 channels (a lane each) of one sequence and walks time in pieces of SCAN_WARPS * SCAN_SEG steps: every
// warp folds its own SCAN_SEG steps into one (E, B) pair  S_out = S_in + (E * S_in + B),  the pairs of the warps before it give its
// S_in, and it walks its steps again for the outputs -- 2 * SCAN_SEG + SCAN_WARPS dependent steps a piece instead of
// SCAN_WARPS * SCAN_SEG, with every warp's loads in flight at once.
constexpr int SCAN_WARPS = 8, SCAN_SEG = 16;

template <typename T>
__global__ void __launch_bounds__(SCAN_WARPS * 32) rglru_scan_kernel(
    const T* __restrict__ proj, int ld, int y_off, const float* __restrict__ y_bias, int x_off,
    const float* __restrict__ x_bias, const int* __restrict__ cu_q, const int* __restrict__ seq_slot,
    const float* __restrict__ a_in, const float* __restrict__ b_in, float* __restrict__ state, float* __restrict__ tail,
    int taps, T* __restrict__ out, int C) {
  let_next_launch_in();   // a product behind this launch may start on its weights
  __shared__ float As[SCAN_WARPS][32], Bs[SCAN_WARPS][32], carry[32];
  const int b = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.y * 32 + lane;
  const int slot = seq_slot[b];
  if (slot < 0) return;
  const bool on = c < C;
  const int n0 = cu_q[b], n1 = cu_q[b + 1];
  if (warp == 0) carry[lane] = on ? state[(size_t)slot * C + c] : 0.f;
  const float yb = on ? y_bias[c] : 0.f;
  __syncthreads();
  for (int t0 = n0; t0 < n1; t0 += SCAN_WARPS * SCAN_SEG) {
    const int first = t0 + warp * SCAN_SEG;
    float av[SCAN_SEG], bv[SCAN_SEG], yv[SCAN_SEG];
#pragma unroll
    for (int i = 0; i < SCAN_SEG; ++i) {
      const int n = first + i;
      const bool ok = on && n < n1;
      av[i] = ok ? a_in[(size_t)n * C + c] : 0.f;      // a - 1; steps behind the end change nothing
      bv[i] = ok ? b_in[(size_t)n * C + c] : 0.f;
      yv[i] = ok ? to_f32<T>(proj[(size_t)n * ld + y_off + c]) : 0.f;
    }
    // with e = a - 1:  S <- S + (e S + b);  two steps (E1, B1) then (e, b) compose to  E = E1 + e + E1 e,  B = B1 + (e B1 + b)
    float E = 0.f, B = 0.f;
#pragma unroll
    for (int i = 0; i < SCAN_SEG; ++i) { B += fmaf(av[i], B, bv[i]); E = fmaf(E, av[i], E + av[i]); }
    As[warp][lane] = E;
    Bs[warp][lane] = B;
    __syncthreads();
    float S = carry[lane];
    for (int w = 0; w < warp; ++w) S += fmaf(As[w][lane], S, Bs[w][lane]);
#pragma unroll
    for (int i = 0; i < SCAN_SEG; ++i) {
      const int n = first + i;
      S += fmaf(av[i], S, bv[i]);
      if (on && n < n1) out[(size_t)n * C + c] = from_f32<T>(S * gelu_tanh_f(yv[i] + yb));
    }
    __syncthreads();          // every warp has read the carry
    if (warp == SCAN_WARPS - 1) carry[lane] = S;
    __syncthreads();
  }
  if (warp != 0 || !on) return;
  state[(size_t)slot * C + c] = carry[lane];
  const int K1 = taps - 1, q = n1 - n0;
  const float xb = x_bias[c];
  for (int j = 0; j < K1; ++j) {   // ascending: an old entry is read before the entry below it is overwritten
    const int idx = q - K1 + j;
    float* dst = tail + ((size_t)slot * K1 + j) * C + c;
    if (idx >= 0) *dst = to_f32<T>(proj[(size_t)(n0 + idx) * ld + x_off + c]) + xb;
    else *dst = tail[((size_t)slot * K1 + j + q) * C + c];
  }
}

template <typename K> int opt_in_smem(K kernel, size_t bytes) {
  if (bytes > 200 * 1024) return DRYFT_ERR_UNSUPPORTED;
  if (bytes > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}
}  // namespace

DRYFT_API int dryft_retention_scan(int is_bf16, const void* proj, int ld, int q_off, int k_off, int v_off, int g_off,
                                   const int* cu_q, const int* seq_slot, const int* tok_pos, const float* inv_freq,
                                   const float* inv_freq_lo, int rot, const double* decay, float* state, void* out, int n_seqs, int H, int dim, int vdim,
                                   float k_scale, float eps, int one_token, int pdl, int early_state, cudaStream_t st) {
  if (n_seqs <= 0) return 0;
  if (H <= 0 || dim <= 0 || vdim <= 0 || rot < 0 || rot > dim || (rot & 1) || H > 65535) return DRYFT_ERR_UNSUPPORTED;
  typedef __nv_bfloat16 bf;
  if (one_token && step_fits(dim, vdim, rot) && ((uintptr_t)state & 15) == 0) {
    const int groups = RT_THREADS / (vdim / 4);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(n_seqs, H);
    cfg.blockDim = dim3(RT_THREADS);
    cfg.dynamicSmemBytes = sizeof(float) * (((size_t)groups * vdim + 2 * (size_t)dim + 3) / 4 * 4 + vdim + rot);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    if (cfg.dynamicSmemBytes <= 48 * 1024) {
      const int rows = step_rows(dim, vdim), early = early_state || !pdl;
      auto run = [&](auto kernel, auto type) {
        typedef decltype(type) T;
        return cudaLaunchKernelEx(&cfg, kernel, (const T*)proj, ld, q_off, k_off, v_off, g_off, seq_slot, tok_pos, inv_freq, inv_freq_lo, rot, decay,
                                  state, (T*)out, H, dim, vdim, k_scale, eps, early);
      };
      const cudaError_t e = is_bf16 ? run(rows <= 4   ? retention_step_kernel<bf, 4>
                                          : rows <= 8 ? retention_step_kernel<bf, 8>
                                                      : retention_step_kernel<bf, STEP_ROWS>, bf())
                                    : run(rows <= 4   ? retention_step_kernel<float, 4>
                                          : rows <= 8 ? retention_step_kernel<float, 8>
                                                      : retention_step_kernel<float, STEP_ROWS>, 0.f);
      return e != cudaSuccess ? (int)e : launch_status();
    }
  }
  const int cols = vdim < RT_THREADS ? vdim : RT_THREADS, groups = RT_THREADS / cols;
  const size_t smem = sizeof(float) * ((size_t)dim * vdim + 2 * (size_t)dim + vdim + (size_t)groups * vdim);
  int rc = is_bf16 ? opt_in_smem(retention_scan_kernel<bf>, smem) : opt_in_smem(retention_scan_kernel<float>, smem);
  if (rc) return rc;
  dim3 grid(n_seqs, H);
  if (is_bf16)
    retention_scan_kernel<bf><<<grid, RT_THREADS, smem, st>>>((const bf*)proj, ld, q_off, k_off, v_off, g_off, cu_q, seq_slot, tok_pos,
                                                              inv_freq, inv_freq_lo, rot, decay, state, (bf*)out, H, dim, vdim, k_scale, eps);
  else
    retention_scan_kernel<float><<<grid, RT_THREADS, smem, st>>>((const float*)proj, ld, q_off, k_off, v_off, g_off, cu_q, seq_slot,
                                                                 tok_pos, inv_freq, inv_freq_lo, rot, decay, state, (float*)out, H, dim, vdim,
                                                                 k_scale, eps);
  return launch_status();
}

// The chunked form: `sbuf` holds (n_tokens / CH + n_seqs) * H * dim * vdim floats, then n_tokens * rot (on an 8-byte boundary:
// one float more).  Four launches.
DRYFT_API int dryft_retention_chunked(int is_bf16, const void* proj, int ld, int q_off, int k_off, int v_off, int g_off,
                                      const int* cu_q, const int* seq_slot, const int* tok_pos, const float* inv_freq,
                                      const float* inv_freq_lo, int rot, const double* decay, float* state, float* sbuf,
                                      void* out, int n_tokens, int n_seqs, int H, int dim, int vdim, float k_scale, float eps,
                                      cudaStream_t st) {
  if (n_seqs <= 0 || n_tokens <= 0) return 0;
  if (H <= 0 || dim <= 0 || vdim <= 0 || vdim > 512 || rot < 0 || rot > dim || (rot & 1) || H > 65535 || n_seqs > 65535)
    return DRYFT_ERR_UNSUPPORTED;
  typedef __nv_bfloat16 bf;
  const int n_chunks = n_tokens / CH + n_seqs;       // an upper bound; blocks behind the last chunk leave at once
  const int dP = (dim + 7) & ~7, vP8 = (vdim + 7) & ~7;
  const size_t smem_a = sizeof(float) * ((size_t)CH * dP + (size_t)CH * vP8 + CH + 1);
  const int dQ = ((dim + 3) & ~3) + 1, vP = (vdim + 3) & ~3;
  const size_t stage = (size_t)CH * (dQ > vP ? dQ : vP);
  const size_t smem_c = sizeof(float) * (stage + (size_t)CH * dQ + (size_t)(CH + 16) * vP + (size_t)CH * (CH + 1) + CH + 1);
  int rc = is_bf16 ? opt_in_smem(retention_chunk_state_kernel<bf>, smem_a) : opt_in_smem(retention_chunk_state_kernel<float>, smem_a);
  if (rc) return rc;
  rc = is_bf16 ? opt_in_smem(retention_chunk_out_kernel<bf>, smem_c) : opt_in_smem(retention_chunk_out_kernel<float>, smem_c);
  if (rc) return rc;
  size_t states = (size_t)n_chunks * H * dim * vdim;
  states += states & 1;
  float2* const angles = reinterpret_cast<float2*>(sbuf + states);
  if (rot > 0) {
    const unsigned blocks = (unsigned)(((size_t)n_tokens * (rot / 2) + 255) / 256);
    retention_angles_kernel<<<blocks, 256, 0, st>>>(tok_pos, inv_freq, inv_freq_lo, angles, n_tokens, rot / 2);
    rc = launch_status();
    if (rc) return rc;
  }
  dim3 grid(n_chunks, H);
  if (is_bf16)
    retention_chunk_state_kernel<bf><<<grid, CK_THREADS, smem_a, st>>>((const bf*)proj, ld, k_off, v_off, cu_q, seq_slot, n_seqs, angles,
                                                                       rot, decay, sbuf, H, dim, vdim, k_scale);
  else
    retention_chunk_state_kernel<float><<<grid, CK_THREADS, smem_a, st>>>((const float*)proj, ld, k_off, v_off, cu_q, seq_slot, n_seqs, angles,
                                                                          rot, decay, sbuf, H, dim, vdim, k_scale);
  int e = launch_status();
  if (e) return e;
  const int per_head = dim * vdim;
  dim3 grid_b(n_seqs, H, (per_head + 255) / 256);
  retention_chunk_prefix_kernel<<<grid_b, 256, 0, st>>>(cu_q, seq_slot, decay, sbuf, state, H, per_head);
  e = launch_status();
  if (e) return e;
  if (is_bf16)
    retention_chunk_out_kernel<bf><<<grid, CK_THREADS, smem_c, st>>>((const bf*)proj, ld, q_off, k_off, v_off, g_off, cu_q, seq_slot, n_seqs,
                                                                     angles, rot, decay, sbuf, (bf*)out, H, dim, vdim, k_scale, eps);
  else
    retention_chunk_out_kernel<float><<<grid, CK_THREADS, smem_c, st>>>((const float*)proj, ld, q_off, k_off, v_off, g_off, cu_q, seq_slot,
                                                                        n_seqs, angles, rot, decay, sbuf,
                                                                        (float*)out, H, dim, vdim, k_scale, eps);
  return launch_status();
}

DRYFT_API int dryft_retention_chunk_tokens() { return CH; }

DRYFT_API int dryft_rglru_gates(int is_bf16, const void* proj, int ld, int x_off, const float* x_bias, const int* tok_slot,
                                const float* conv_w, const float* conv_b, int taps, const float* tail, const float* w_gates,
                                const float* b_a, const float* b_i, const float* sp_lam, float c_mult, float* a_out, float* b_out,
                                int n_tokens, int C, int n_blocks, cudaStream_t st) {
  if (n_tokens <= 0) return 0;
  if (taps < 1 || n_blocks < 1 || C % n_blocks || n_blocks > 65535) return DRYFT_ERR_UNSUPPORTED;
  typedef __nv_bfloat16 bf;
  const int nb = C / n_blocks;
  const size_t smem = sizeof(float) * (size_t)GT * nb;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long blocks = (long long)((n_tokens + GT - 1) / GT) * n_blocks, few_blocks = blocks * ((nb + FEW_COLS - 1) / FEW_COLS);
  if (few_blocks <= (long long)FEW_BLOCKS_PER_SM * sms && few_smem(GT, nb) <= 96 * 1024) {
    const int vec = nb % 4 == 0 && ((uintptr_t)w_gates & 15) == 0;
#define DRYFT_FEW(TT, NT)                                                                                                             \
  do {                                                                                                                               \
    const int rc = opt_in_smem(rglru_gates_few_kernel<TT, NT>, few_smem(NT, nb) + 2048 /* `logits` */);                              \
    if (rc) return rc;                                                                                                               \
    rglru_gates_few_kernel<TT, NT><<<dim3((n_tokens + NT - 1) / NT, n_blocks, (nb + FEW_COLS - 1) / FEW_COLS), G_THREADS,            \
                                     few_smem(NT, nb), st>>>((const TT*)proj, ld, x_off, x_bias, tok_slot, conv_w, conv_b, taps,     \
                                                             tail, w_gates, b_a, b_i, sp_lam, c_mult, a_out, b_out, n_tokens, C, nb, \
                                                             vec);                                                                   \
  } while (0)
#define DRYFT_FEW_BY_TOKENS(TT)                  \
  do {                                           \
    if (n_tokens == 1) DRYFT_FEW(TT, 1);         \
    else if (n_tokens == 2) DRYFT_FEW(TT, 2);    \
    else if (n_tokens <= 4) DRYFT_FEW(TT, 4);    \
    else DRYFT_FEW(TT, 8);                       \
  } while (0)
    if (is_bf16) DRYFT_FEW_BY_TOKENS(bf);
    else DRYFT_FEW_BY_TOKENS(float);
#undef DRYFT_FEW_BY_TOKENS
#undef DRYFT_FEW
    return launch_status();
  }
  // groups beside one another halve the blocks: worth it once all of them do not run at once any more (four a multiprocessor; 16 gate
  // blocks of 128, 512 blocks: 24.9 us without and 26.6 with, 768 blocks: 43 and 32)
  const int groups = nb >= G_THREADS || blocks <= 4LL * sms ? 1 : G_THREADS / nb < 4 ? G_THREADS / nb : 4;
  const bool ahead = blocks <= 2LL * sms;
  const size_t many = smem * groups;
  dim3 grid((n_tokens + GT * groups - 1) / (GT * groups), n_blocks);
#define DRYFT_MANY(TT, AHEAD)                                                                                                          \
  do {                                                                                                                               \
    const int rc = opt_in_smem(rglru_gates_kernel<TT, AHEAD>, many);                                                                 \
    if (rc) return rc;                                                                                                               \
    rglru_gates_kernel<TT, AHEAD><<<grid, G_THREADS, many, st>>>((const TT*)proj, ld, x_off, x_bias, tok_slot, conv_w, conv_b, taps,  \
                                                                 tail, w_gates, b_a, b_i, sp_lam, c_mult, a_out, b_out, n_tokens, C, \
                                                                 nb, groups);                                                        \
  } while (0)
  if (is_bf16 && ahead) DRYFT_MANY(bf, true);
  else if (is_bf16) DRYFT_MANY(bf, false);
  else if (ahead) DRYFT_MANY(float, true);
  else DRYFT_MANY(float, false);
#undef DRYFT_MANY
  return launch_status();
}

DRYFT_API int dryft_rglru_scan(int is_bf16, const void* proj, int ld, int y_off, const float* y_bias, int x_off,
                               const float* x_bias, const int* cu_q, const int* seq_slot, const float* a_in, const float* b_in,
                               float* state, float* tail, int taps, void* out, int n_seqs, int C, cudaStream_t st) {
  if (n_seqs <= 0) return 0;
  typedef __nv_bfloat16 bf;
  const int threads = SCAN_WARPS * 32;
  dim3 grid(n_seqs, (C + 31) / 32);
  if (grid.y > 65535) return DRYFT_ERR_UNSUPPORTED;
  if (is_bf16)
    rglru_scan_kernel<bf><<<grid, threads, 0, st>>>((const bf*)proj, ld, y_off, y_bias, x_off, x_bias, cu_q, seq_slot, a_in, b_in, state,
                                                    tail, taps, (bf*)out, C);
  else
    rglru_scan_kernel<float><<<grid, threads, 0, st>>>((const float*)proj, ld, y_off, y_bias, x_off, x_bias, cu_q, seq_slot, a_in, b_in,
                                                       state, tail, taps, (float*)out, C);
  return launch_status();
}
