// A state-space mixer whose decay differs per channel and per entry of the state (selective scan):
//
//   S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n        A = -exp(A_log), dt = softplus(dt_pre + dt_bias)
//   y_c      = sum_n S[c, n] C_n + D_c x_c,   out_c = y_c * silu(z_c)
//
// x, z and dt_pre have one number per channel and token, B and C one per state entry and token (shared by
// all channels).  S [channels, N] per request is 32-bit, starts at zero and is carried from token to token;
// everything here is 32-bit, the output is rounded once for the output projection.
//
// Kernels: the causal convolution of x with the request's last inputs kept between steps (+ SiLU), and
// the walk, of which there are three: states of up to 16 entries an entry a lane, in one piece; steps of single
// tokens of such states; larger states, and such of few channels and many tokens, a share of the entries a lane, in segments.  The walk is sequential in
// tokens; a CTA takes some channels of one request, WL lanes a channel,
// each lane a share of the state's entries in registers.  A chunk of tokens waits in shared memory while the
// next one arrives there (cp.async); step sizes are formed once per channel and token before the chunk is
// walked.  From token to token passes only the state's own update: every lane leaves its share of the sum
// over the state in shared memory, and the sums, the skip term and the gate are formed after the chunk, a
// thread per channel and token.
//
// A long portion is there cut into segments of tokens that are walked side by side, in two launches: the first walks every
// segment but the last from zeros (the first one from the request's state) for its closing state and the sum of its
// step sizes, the second takes every segment again from its opening state, which follows from the segments before it
// (S <- exp(A sum dt) S + S_segment), and leaves the outputs.  Everything stays 32-bit; the errors against 64-bit are
// those of the walk in one piece.
#include "common.cuh"

namespace {
constexpr int kThreads = 256;

__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// ---- causal convolution over the last `taps` inputs of every channel, then SiLU -------------------
struct ConvParams {
  const float* proj;     // [tokens, ld]; the convolution's inputs at columns [conv_at, conv_at + channels)
  int ld, conv_at, channels, taps;
  float* kept;           // [slots, taps - 1, channels]: the request's last inputs, oldest first
  const int* row_req;
  const int* q_start;
  const int* state_slot;
  int n_slots;
};

// grid (rows, blocks of channels).  out32 [tokens, channels] floats; out_t the same rounded to T (or null).
template <typename T>
__global__ void __launch_bounds__(kThreads) conv_silu_kernel(float* __restrict__ out32, T* __restrict__ out_t,
                                                             const T* __restrict__ taps_w, const T* __restrict__ taps_b,
                                                             ConvParams p) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, r = p.row_req[t], first = p.q_start[r], slot = p.state_slot[r];
  const int K = p.taps, C = p.channels;
  const int c = blockIdx.y * kThreads + threadIdx.x;
  if (c >= C) return;
  if (slot == -1) {       // a row of padding
    out32[(size_t)t * C + c] = 0.f;
    if (out_t != nullptr) out_t[(size_t)t * C + c] = from_f32<T>(0.f);
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  const float* kept = p.kept + (size_t)slot * (K - 1) * C;
  float acc = to_f32(taps_b[c]);
  for (int jj = 0; jj < K; ++jj) {
    const int src = t - (K - 1) + jj;       // the last tap meets the row itself
    const float u = src >= first ? p.proj[(size_t)src * p.ld + p.conv_at + c]
                                 : kept[(size_t)((K - 1) + (src - first)) * C + c];
    acc = fmaf(to_f32(taps_w[(size_t)c * K + jj]), u, acc);
  }
  const float v = silu_f(acc);
  out32[(size_t)t * C + c] = v;
  if (out_t != nullptr) out_t[(size_t)t * C + c] = from_f32<T>(v);
}

// The same for four taps and many rows: a thread takes CONV_ROWS neighbouring rows of its channel, whose inputs are asked
// for at once and serve up to four rows each.  Bound by what it reads and writes (one input, 6 bytes out a channel and
// row); 2,048 x 1,792 in 17 us (25 a thread a row), 608 x 3,072 in 11.6 (13.7).
constexpr int CONV_ROWS = 8;
template <typename T>
__global__ void __launch_bounds__(kThreads) conv_silu4_kernel(float* __restrict__ out32, T* __restrict__ out_t,
                                                              const T* __restrict__ taps_w, const T* __restrict__ taps_b,
                                                              ConvParams p, int tokens) {
  pdl_trigger();
  pdl_wait();
  const int t0 = blockIdx.x * CONV_ROWS, C = p.channels;
  const int c = blockIdx.y * kThreads + threadIdx.x;
  if (c >= C) return;
  float u[CONV_ROWS + 3], w[4];
#pragma unroll
  for (int i = 0; i < CONV_ROWS + 3; ++i) {
    const int src = t0 - 3 + i;
    u[i] = src >= 0 && src < tokens ? p.proj[(size_t)src * p.ld + p.conv_at + c] : 0.f;
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = to_f32(taps_w[(size_t)c * 4 + j]);
  const float bias = to_f32(taps_b[c]);
#pragma unroll
  for (int i = 0; i < CONV_ROWS; ++i) {
    const int t = t0 + i;
    if (t >= tokens) break;
    const int r = p.row_req[t], first = p.q_start[r], slot = p.state_slot[r];
    float v = 0.f;            // a row of padding
    if (slot != -1) {
      if (slot < 0 || slot >= p.n_slots) {
        lab_set_error(LAB_ERR_PAGE_RANGE);
        continue;
      }
      float acc = bias;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int src = t - 3 + j;
        acc = fmaf(w[j], src >= first ? u[i + j] : p.kept[((size_t)slot * 3 + (3 + src - first)) * C + c], acc);
      }
      v = silu_f(acc);
    }
    out32[(size_t)t * C + c] = v;
    if (out_t != nullptr) out_t[(size_t)t * C + c] = from_f32<T>(v);
  }
}

// grid (requests, blocks of channels), after every row of the step has read the kept inputs.  A thread walks
// the kept rows of its one channel oldest first: what it overwrites it has already moved.
__global__ void __launch_bounds__(kThreads) conv_keep_inputs_kernel(ConvParams p) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  const int first = p.q_start[r], n = p.q_start[r + 1] - first, slot = p.state_slot[r];
  if (n <= 0 || slot == -1) return;
  if (slot < 0 || slot >= p.n_slots) {
    if (threadIdx.x == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  const int K1 = p.taps - 1, C = p.channels;
  float* kept = p.kept + (size_t)slot * K1 * C;
  const int c = blockIdx.y * kThreads + threadIdx.x;
  if (c >= C) return;
  for (int i = 0; i < K1; ++i) {
    const int s = n - K1 + i;               // the step's row that becomes kept row i
    kept[(size_t)i * C + c] = s >= 0 ? p.proj[(size_t)(first + s) * p.ld + p.conv_at + c] : kept[(size_t)(i + n) * C + c];
  }
}

// ---- the walk ----------------------------------------------------------------------------------------
constexpr int WT = 32;        // tokens a chunk
constexpr int WTHREADS = 128;
constexpr int SCAN_MAX_STATE = 256;
constexpr int LONG_WALK = 256;      // tokens from which the next kernel is let in at the walk's end only

// What may be moved 16 bytes at a time: rows of dt_pre, x and z; of B and C; the state's; the output's.
enum { VEC_ROWS = 1, VEC_BC = 2, VEC_STATE = 4, VEC_OUT = 8 };
struct ScanParams {
  const float* x;        // [tokens, ld_x] after the convolution and SiLU
  const float* dt_pre;   // [tokens, ld_dt] the step sizes before bias and softplus
  const float* bc;       // [tokens, ld_bc]: B at columns [b_at, b_at + N), C at [c_at, c_at + N)
  const float* z;        // [tokens, ld_z] the gate's input
  float* state;          // [slots, channels, N]
  const int* q_start;
  const int* state_slot;
  int ld_x, ld_dt, ld_bc, ld_z, b_at, c_at, channels, N, n_slots, write, ld_out;
  int vec;               // rows of all inputs may be copied 16 bytes at a time; the walks of small states: VEC_ bits (more
                         // fields change the other walk's registers: 2,048 tokens, 768 channels of 128 entries 367 us, not 333)
  int segments;          // a request's rows are cut into at most that many segments of whole chunks
  float* states;         // [requests, segments, channels, N]: 0, a copy of the request's state; i, the state at the end
                         // of segment i - 1 (from zeros, of segment 0 from the request's state)
  float* sums;           // [requests, segments, channels]: the sum of the step sizes of segment i - 1
};
// What a launch of the walk does: everything in one piece, the segments' closing states, or the outputs.
enum { SCAN_WHOLE, SCAN_CLOSE, SCAN_OUTPUT };

// 4 or 16 bytes from global to shared memory without a register in between; waited for by cp_async_wait_all.
__device__ __forceinline__ void cp_async_f32(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_f32x4(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The library's exponential: a slow decay's error comes with the same sign at every token and adds up over the state's
// memory, so a form that is off by more is none.  (One by a range reduction and a polynomial, two entries an instruction,
// took the mixer 242 us for 2,048 tokens, this one 222.)
__device__ __forceinline__ f32x2 exp_of(f32x2 x) { return pair_of(expf(low_of(x)), expf(high_of(x))); }

// The first `n` of two entries, zeros for the others.
__device__ __forceinline__ f32x2 first_of(f32x2 v, int n) { return n >= 2 ? v : n == 1 ? v & 0xffffffffull : 0ull; }

// Floats of one chunk's inputs as they arrive: dt_pre, x, z [WT][channels] each, then B and C [WT][N4] each, N4 the
// state's entries in whole quads.
__host__ __device__ inline int scan_chunk_floats(int wc, int n4) { return 3 * WT * wc + 2 * WT * n4; }

// Lane l of a channel's WL holds the quads l, l + WL, ... of its state, R entries in all.  What bounds the walk, once
// there are CTAs enough, is the issue of instructions: most of an entry's and token's are its exponential's, the others
// take two entries each; a token of a CTA also takes its step sizes, gates and copies.  Measured on a B200, inputs from
// memory, 1,792 channels of 16 entries, before those had a walk of their own: 8 requests of 250 tokens 82 us (115 with eight lanes a channel and an entry an
// instruction); one of 2,048 129 us in eleven segments (352 in one piece of that form), issuing in two cycles of three.
// QUADS: the state is whole quads; else the entries that fill the last one are kept at zero (an infinite step would leave
// no numbers there).
template <typename T, int WL, int R, int MODE, bool QUADS>
__global__ void __launch_bounds__(WTHREADS) selective_scan_kernel(T* __restrict__ out, const T* __restrict__ a_log,
                                                                  const T* __restrict__ skip,
                                                                  const T* __restrict__ dt_bias, ScanParams p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int WC = WTHREADS / WL, Q = R / 4;
  const int N = p.N, n4 = (N + 3) & ~3, chunk_floats = scan_chunk_floats(WC, n4);
  float* s_in = smem;                          // two chunks of inputs: one walked, one arriving
  float* s_dx = smem + 2 * chunk_floats;       // [WT][WC] step size times x
  float* s_part = s_dx + WT * WC;              // [WT][WC][WL] every lane's share of the sum over the state
  pdl_wait();
  const int r = blockIdx.y, c0 = blockIdx.x * WC;
  int first = p.q_start[r], n = p.q_start[r + 1] - first;
  const int slot = p.state_slot[r];
  int seg = 0, last = 0;      // this CTA's segment, the request's last one
  if (MODE != SCAN_WHOLE && n > 0) {
    const int len = (((n + p.segments - 1) / p.segments) + WT - 1) / WT * WT;
    seg = blockIdx.z;
    last = (n - 1) / len;
    if (MODE == SCAN_CLOSE && seg >= last) return;
    first += seg * len;
    n = min(len, n - seg * len);
  }
  if (MODE == SCAN_WHOLE && n < LONG_WALK) pdl_trigger();
  if (n <= 0) return;
  const int tid = threadIdx.x, ch = tid / WL, l = tid % WL, c = c0 + ch;
  const bool live = c < p.channels;
  if (MODE == SCAN_CLOSE && (slot < 0 || slot >= p.n_slots)) return;      // (the next launch deals with these)
  if (slot == -1) {       // rows of padding leave zeros
    for (int i = tid; i < n * WC; i += WTHREADS)
      if (c0 + i % WC < p.channels) out[(size_t)(first + i / WC) * p.ld_out + c0 + i % WC] = from_f32<T>(0.f);
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  if (!QUADS) {      // the last quad's missing entries of B and C are zeros, which no copy touches
    for (int i = tid; i < 2 * chunk_floats; i += WTHREADS) s_in[i] = 0.f;
    __syncthreads();
  }
  // a chunk's inputs set out for shared memory; channels beyond the last read nothing and stay unused
  auto fetch = [&](int t0, float* buf) {
    const int nt = min(WT, n - t0);
    float *b_dt = buf, *b_x = buf + WT * WC, *b_z = buf + 2 * WT * WC, *b_b = buf + 3 * WT * WC, *b_c = b_b + WT * n4;
    const size_t row0 = (size_t)(first + t0);
    if (p.vec) {
      for (int i = tid; i < nt * (WC / 4); i += WTHREADS) {
        const int cc = c0 + 4 * (i % (WC / 4));
        if (cc >= p.channels) continue;
        const size_t row = row0 + i / (WC / 4);
        cp_async_f32x4(b_dt + 4 * i, p.dt_pre + row * p.ld_dt + cc);
        cp_async_f32x4(b_x + 4 * i, p.x + row * p.ld_x + cc);
        if (MODE != SCAN_CLOSE) cp_async_f32x4(b_z + 4 * i, p.z + row * p.ld_z + cc);
      }
      for (int i = tid; i < nt * (n4 / 4); i += WTHREADS) {
        const float* row = p.bc + (row0 + i / (n4 / 4)) * p.ld_bc + 4 * (i % (n4 / 4));
        cp_async_f32x4(b_b + 4 * i, row + p.b_at);
        if (MODE != SCAN_CLOSE) cp_async_f32x4(b_c + 4 * i, row + p.c_at);
      }
      return;
    }
    for (int i = tid; i < nt * WC; i += WTHREADS) {
      const int cc = c0 + i % WC;
      if (cc >= p.channels) continue;
      const size_t row = row0 + i / WC;
      cp_async_f32(b_dt + i, p.dt_pre + row * p.ld_dt + cc);
      cp_async_f32(b_x + i, p.x + row * p.ld_x + cc);
      if (MODE != SCAN_CLOSE) cp_async_f32(b_z + i, p.z + row * p.ld_z + cc);
    }
    for (int i = tid; i < nt * N; i += WTHREADS) {
      const float* row = p.bc + (row0 + i / N) * p.ld_bc + i % N;
      cp_async_f32(b_b + i / N * n4 + i % N, row + p.b_at);
      if (MODE != SCAN_CLOSE) cp_async_f32(b_c + i / N * n4 + i % N, row + p.c_at);
    }
  };
  fetch(0, s_in);
  auto entry = [&](int i) { return ((i / 4) * WL + l) * 4 + i % 4; };      // the state's entry that S[i] holds
  float S[R], A[R];
  float* st = p.state + ((size_t)slot * p.channels + (live ? c : 0)) * N;
  const size_t per_segment = (size_t)p.channels * N;
  float* kept = MODE == SCAN_WHOLE ? nullptr : p.states + (size_t)r * p.segments * per_segment + (size_t)(live ? c : 0) * N;
  const float* sums = MODE == SCAN_WHOLE ? nullptr : p.sums + (size_t)r * p.segments * p.channels + (live ? c : 0);
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int e = entry(i);
    const bool has = live && e < N;
    A[i] = has ? -expf(to_f32(a_log[(size_t)c * N + e])) : 0.f;
    S[i] = 0.f;
    if (!has) continue;
    if (MODE == SCAN_WHOLE || (MODE == SCAN_OUTPUT && last == 0)) {
      S[i] = st[e];
    } else if (MODE == SCAN_CLOSE) {
      // (the last segment's CTA of the next launch writes the request's state while others still open theirs)
      if (seg == 0) kept[e] = S[i] = st[e];
    } else {
      S[i] = kept[(seg == 0 ? 0 : per_segment) + e];
    }
  }
  if (MODE == SCAN_OUTPUT) {
    for (int g = 2; g <= seg; ++g) {
      const float dt = sums[(size_t)g * p.channels];
#pragma unroll
      for (int i = 0; i < R; ++i)
        if (live && entry(i) < N) S[i] = fmaf(expf(dt * A[i]), S[i], kept[g * per_segment + entry(i)]);
    }
  }
  f32x2 S2[R / 2], A2[R / 2];
#pragma unroll
  for (int i = 0; i < R / 2; ++i) S2[i] = pair_of(S[2 * i], S[2 * i + 1]), A2[i] = pair_of(A[2 * i], A[2 * i + 1]);
  float dt_sum = 0.f;      // SCAN_CLOSE: of channel tid % WC, over this thread's tokens
  int which = 0;
  for (int t0 = 0; t0 < n; t0 += WT, which ^= 1) {
    const int nt = min(WT, n - t0);
    float* buf = s_in + which * chunk_floats;
    float *b_dt = buf, *b_x = buf + WT * WC, *b_z = buf + 2 * WT * WC, *b_b = buf + 3 * WT * WC, *b_c = b_b + WT * n4;
    cp_async_wait_all();
    __syncthreads();       // the chunk is here; the chunk before has been written out, its buffer is free
    if (t0 + WT < n) fetch(t0 + WT, s_in + (which ^ 1) * chunk_floats);
    // step sizes once per channel and token
    for (int i = tid; i < nt * WC; i += WTHREADS) {
      const int cc = c0 + i % WC;
      float dt = 0.f, dx = 0.f;
      if (cc < p.channels) {
        dt = softplus_f(b_dt[i] + to_f32(dt_bias[cc]));
        dx = dt * b_x[i];
      }
      b_dt[i] = dt;
      s_dx[i] = dx;
      if (MODE == SCAN_CLOSE) dt_sum += dt;
    }
    __syncthreads();
    // the walk: nothing but the state's own update passes from token to token (with few entries a lane four tokens in flight: one
    // request of 2,048 tokens in segments 129 us, 131 by two; no gain with more)
#pragma unroll (R == 4 ? 4 : 2)
    for (int tt = 0; tt < nt; ++tt) {
      const float dt = b_dt[tt * WC + ch], dx = s_dx[tt * WC + ch];
      const f32x2 dt2 = pair_of(dt, dt), dx2 = pair_of(dx, dx);
      f32x2 acc = 0ull;      // two zeros
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int e = (q * WL + l) * 4;
        if (Q * WL * 4 > 16 && e >= n4) break;
        if (Q * WL * 4 == 16 && e >= n4) continue;
        const ulonglong2 bq = *reinterpret_cast<const ulonglong2*>(b_b + tt * n4 + e);
        S2[2 * q] = fma2(exp_of(mul2(dt2, A2[2 * q])), S2[2 * q], mul2(dx2, bq.x));
        S2[2 * q + 1] = fma2(exp_of(mul2(dt2, A2[2 * q + 1])), S2[2 * q + 1], mul2(dx2, bq.y));
        if (!QUADS) S2[2 * q] = first_of(S2[2 * q], N - e), S2[2 * q + 1] = first_of(S2[2 * q + 1], N - e - 2);
        if (MODE != SCAN_CLOSE) {
          const ulonglong2 cq = *reinterpret_cast<const ulonglong2*>(b_c + tt * n4 + e);
          acc = fma2(S2[2 * q], cq.x, acc);
          acc = fma2(S2[2 * q + 1], cq.y, acc);
        }
      }
      if (MODE != SCAN_CLOSE) s_part[tt * WTHREADS + tid] = low_of(acc) + high_of(acc);
    }
    if (MODE == SCAN_CLOSE) continue;
    __syncthreads();
    // the sum over the lanes (in their order), the skip term and the gate, a thread per channel and token
    for (int i = tid; i < nt * WC; i += WTHREADS) {
      const int cc = c0 + i % WC;
      if (cc >= p.channels) continue;
      float4 sum = *reinterpret_cast<const float4*>(s_part + (size_t)i * WL);
      if (WL == 8) {
        const float4 hi = *reinterpret_cast<const float4*>(s_part + (size_t)i * WL + 4);
        sum.x += hi.x, sum.y += hi.y, sum.z += hi.z, sum.w += hi.w;
      }
      const float acc = (sum.x + sum.z) + (sum.y + sum.w);
      out[(size_t)(first + t0 + i / WC) * p.ld_out + cc] =
          from_f32<T>(fmaf(to_f32(skip[cc]), b_x[i], acc) * silu_f(b_z[i]));
    }
  }
  pdl_trigger();      // (not earlier: the next kernel's blocks would settle beside this one's and slow them down)
  if (MODE == SCAN_CLOSE) {
    s_part[tid] = dt_sum;      // WC threads apart: the same channel
    __syncthreads();
    if (tid < WC && c0 + tid < p.channels) {
      float all = 0.f;
#pragma unroll
      for (int i = 0; i < WTHREADS / WC; ++i) all += s_part[i * WC + tid];
      p.sums[((size_t)r * p.segments + seg + 1) * p.channels + c0 + tid] = all;
    }
  }
  float* to = MODE == SCAN_CLOSE ? kept + (seg + 1) * per_segment : st;
  if (live && (MODE == SCAN_CLOSE || (p.write && seg == last))) {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (entry(i) < N) to[entry(i)] = i % 2 == 0 ? low_of(S2[i / 2]) : high_of(S2[i / 2]);
  }
}

// ---- the walk of states of up to 16 entries ----------------------------------------------------------
// A lane an entry: LN lanes a channel, 32 / LN channels a warp.  A warp forms its channels' step sizes for a chunk of WTS
// tokens, walks it, and forms its channels' outputs; only the chunk's inputs, brought by cp.async, are shared by the CTA's
// warps, so they meet once a chunk.  Inputs lie so that a lane reads four tokens at a time; every lane leaves its
// share of the sum over the state in shared memory.  A request's rows are walked in one piece: its numbers depend on neither
// the cut nor the batch.
// What bounds it: the issue of instructions, most of them the exponential's, by the few warps that a request's channels make
// (six a multiprocessor for 1,792 channels of 16; they issue in two cycles of five).  The mixer around it (us, from a graph)
// against four entries a lane, in segments from 320 tokens on: 1,792 channels, one request of 2,048 tokens 212 (220), of 700
// 110 (121), of 319 75 (113), eight of 250 157 (172); 3,072 channels, 1,500 tokens 219 (257).
constexpr int SMALL_STATE = 16;
struct ScanTile {      // floats of shared memory
  int in, chunk, dt, part, out, total;
  __host__ __device__ ScanTile(int wc, int ln, int wts, int warps) {
    chunk = 3 * wts * wc + 2 * wts * ln;            // dt_pre, x, z [wts][wc], then B and C [wts][ln]
    in = 0;
    dt = 2 * chunk;                                 // step sizes and step size times x, [wc][wts + 4] each
    part = dt + 2 * wc * (wts + 4);                 // [warp][wts][36]
    out = part + warps * wts * 36;                  // two chunks of [wts][wc]
    total = out + 2 * wts * wc;
  }
};

template <typename T, int LN, int WARPS, int WTS, bool WHOLE_LANES>
__global__ void __launch_bounds__(32 * WARPS) selective_walk_kernel(T* __restrict__ out, const T* __restrict__ a_log,
                                                                    const T* __restrict__ skip,
                                                                    const T* __restrict__ dt_bias, ScanParams p) {
  constexpr int THREADS = 32 * WARPS, CPW = 32 / LN, WC = WARPS * CPW, LD = WTS + 4, SL = 36;
  static_assert(WTS % 4 == 0, "four tokens at a time");
  extern __shared__ __align__(16) float smem[];
  const ScanTile tile(WC, LN, WTS, WARPS);
  pdl_wait();
  const int r = blockIdx.y, c0 = blockIdx.x * WC, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int first = p.q_start[r], n = p.q_start[r + 1] - first, slot = p.state_slot[r];
  if (n < LONG_WALK) pdl_trigger();
  if (n <= 0) return;
  if (slot == -1) {       // rows of padding leave zeros
    for (int i = tid; i < n * WC; i += THREADS)
      if (c0 + i % WC < p.channels) out[(size_t)(first + i / WC) * p.ld_out + c0 + i % WC] = from_f32<T>(0.f);
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  const int N = WHOLE_LANES ? LN : p.N;
  // a chunk's inputs set out for shared memory; channels and entries beyond the last read nothing and stay unused
  auto fetch = [&](int t0, float* buf) {
    const int nt = min(WTS, n - t0);
    const size_t row0 = (size_t)(first + t0);
    float *b_x = buf + WTS * WC, *b_z = b_x + WTS * WC, *b_b = b_z + WTS * WC, *b_c = b_b + WTS * LN;
    if (p.vec & VEC_ROWS) {
      for (int i = tid; i < nt * (WC / 4); i += THREADS) {
        const int cc = c0 + 4 * (i % (WC / 4));
        if (cc >= p.channels) continue;
        const size_t row = row0 + i / (WC / 4);
        cp_async_f32x4(buf + 4 * i, p.dt_pre + row * p.ld_dt + cc);
        cp_async_f32x4(b_x + 4 * i, p.x + row * p.ld_x + cc);
        cp_async_f32x4(b_z + 4 * i, p.z + row * p.ld_z + cc);
      }
    } else {
      for (int i = tid; i < nt * WC; i += THREADS) {
        const int cc = c0 + i % WC;
        if (cc >= p.channels) continue;
        const size_t row = row0 + i / WC;
        cp_async_f32(buf + i, p.dt_pre + row * p.ld_dt + cc);
        cp_async_f32(b_x + i, p.x + row * p.ld_x + cc);
        cp_async_f32(b_z + i, p.z + row * p.ld_z + cc);
      }
    }
    if (p.vec & VEC_BC) {
      for (int i = tid; i < nt * (N / 4); i += THREADS) {
        const int e = 4 * (i % (N / 4)), t = i / (N / 4);
        const float* row = p.bc + (row0 + t) * p.ld_bc + e;
        cp_async_f32x4(b_b + t * LN + e, row + p.b_at);
        cp_async_f32x4(b_c + t * LN + e, row + p.c_at);
      }
      return;
    }
    for (int i = tid; i < nt * N; i += THREADS) {
      const int e = i % N, t = i / N;
      const float* row = p.bc + (row0 + t) * p.ld_bc + e;
      cp_async_f32(b_b + t * LN + e, row + p.b_at);
      cp_async_f32(b_c + t * LN + e, row + p.c_at);
    }
  };
  fetch(0, smem);
  const int ch = lane / LN, e = lane % LN, mine = warp * CPW + ch, c = c0 + mine;      // this lane's channel and entry
  const bool has = c < p.channels && e < N;
  const float A = has ? -expf(to_f32(a_log[(size_t)c * N + e])) : 0.f;
  float* st = p.state + ((size_t)slot * p.channels + (has ? c : 0)) * N + e;
  float S = has ? *st : 0.f;
  // what the tokens' terms take: lane l is at token l / CPW (+ 32 / CPW, ...) of channel l % CPW of the warp's
  const int tc = lane % CPW, of = warp * CPW + tc;
  const bool term = c0 + of < p.channels;
  const float bias = term ? to_f32(dt_bias[c0 + of]) : 0.f, D = term ? to_f32(skip[c0 + of]) : 0.f;
  float *s_dt = smem + tile.dt, *s_dx = s_dt + WC * LD, *s_part = smem + tile.part + warp * WTS * SL;
  T* s_out = reinterpret_cast<T*>(smem + tile.out);
  // outputs of a chunk, row by row
  auto leave = [&](int t0, int which) {
    const int nt = min(WTS, n - t0);
    const T* from = s_out + which * WTS * WC;
    constexpr int UNIT = 16 / (int)sizeof(T), PER = WC / UNIT;
    if (PER > 0 && (p.vec & VEC_OUT)) {
      for (int i = tid; i < nt * PER; i += THREADS) {
        const int cc = c0 + UNIT * (i % (PER > 0 ? PER : 1)), t = i / (PER > 0 ? PER : 1);
        if (cc < p.channels)
          *reinterpret_cast<uint4*>(out + (size_t)(first + t0 + t) * p.ld_out + cc) = *reinterpret_cast<const uint4*>(from + UNIT * i);
      }
      return;
    }
    for (int i = tid; i < nt * WC; i += THREADS)
      if (c0 + i % WC < p.channels) out[(size_t)(first + t0 + i / WC) * p.ld_out + c0 + i % WC] = from[i];
  };
  int which = 0;
  for (int t0 = 0; t0 < n; t0 += WTS, which ^= 1) {
    const int nt = min(WTS, n - t0);
    const float* buf = smem + which * tile.chunk;
    const float *b_x = buf + WTS * WC, *b_z = b_x + WTS * WC, *b_b = b_z + WTS * WC, *b_c = b_b + WTS * LN;
    cp_async_wait_all();
    __syncthreads();       // the chunk is here, every warp is done with the one before
    if (t0 + WTS < n) fetch(t0 + WTS, smem + (which ^ 1) * tile.chunk);
    if (t0 > 0) leave(t0 - WTS, which ^ 1);
#pragma unroll
    for (int i = 0; i < (CPW * WTS + 31) / 32; ++i) {
      const int t = min((lane + 32 * i) / CPW, WTS - 1);      // (a chunk of few tokens: several lanes form the last one's)
      const float dt = term ? softplus_f(buf[t * WC + of] + bias) : 0.f;      // (tokens beyond the last: never read)
      s_dt[of * LD + t] = dt;
      s_dx[of * LD + t] = dt * b_x[t * WC + of];
    }
    __syncwarp();
    const float *my_dt = s_dt + mine * LD, *my_dx = s_dx + mine * LD, *my_b = b_b + e, *my_c = b_c + e;
    auto token = [&](float decay, float dx, float b) {
      S = fmaf(decay, S, dx * b);
      if (!WHOLE_LANES) S = has ? S : 0.f;      // (an infinite step would leave no number)
    };
    // LOT tokens at a time: only the state's own update passes from one to the next
    constexpr int LOT = 8;
    int t = 0;
    for (; t + LOT <= nt; t += LOT) {
      float dt[LOT], dx[LOT], b[LOT], cc[LOT];
#pragma unroll
      for (int i = 0; i < LOT; i += 4) {
        const float4 q = load4(my_dt + t + i), x = load4(my_dx + t + i);
        dt[i] = q.x, dt[i + 1] = q.y, dt[i + 2] = q.z, dt[i + 3] = q.w;
        dx[i] = x.x, dx[i + 1] = x.y, dx[i + 2] = x.z, dx[i + 3] = x.w;
      }
#pragma unroll
      for (int i = 0; i < LOT; ++i) b[i] = my_b[(t + i) * LN], cc[i] = my_c[(t + i) * LN];
#pragma unroll
      for (int i = 0; i < LOT; ++i) dt[i] = expf(dt[i] * A);
#pragma unroll
      for (int i = 0; i < LOT; ++i) {
        token(dt[i], dx[i], b[i]);
        cc[i] = WHOLE_LANES || has ? S * cc[i] : 0.f;
      }
#pragma unroll
      for (int i = 0; i < LOT; ++i) s_part[(t + i) * SL + lane] = cc[i];
    }
    for (; t < nt; ++t) {
      token(expf(my_dt[t] * A), my_dx[t], my_b[t * LN]);
      s_part[t * SL + lane] = WHOLE_LANES || has ? S * my_c[t * LN] : 0.f;
    }
    __syncwarp();
    // the sum over the lanes (in their order), the skip term and the gate
#pragma unroll
    for (int i = 0; i < (CPW * WTS + 31) / 32; ++i) {
      const int t = (lane + 32 * i) / CPW;
      if (!term || t >= nt) continue;
      const float* from = s_part + t * SL + tc * LN;
      float4 sum = load4(from);
#pragma unroll
      for (int q = 1; q < LN / 4; ++q) {
        const float4 v = load4(from + 4 * q);
        sum.x += v.x, sum.y += v.y, sum.z += v.z, sum.w += v.w;
      }
      const float acc = (sum.x + sum.z) + (sum.y + sum.w);
      s_out[which * WTS * WC + t * WC + of] = from_f32<T>(fmaf(D, b_x[t * WC + of], acc) * silu_f(b_z[t * WC + of]));
    }
    __syncwarp();
  }
  pdl_trigger();      // (not earlier: the next kernel's blocks would settle beside this one's and slow them down)
  __syncthreads();
  leave((n - 1) / WTS * WTS, which ^ 1);
  if (has && p.write) *st = S;
}

// A step of single tokens: a thread four entries of a channel, QL threads a channel, everything straight from memory.  The
// same sums in the same order as the walk's.  Bound by the state's way from and to memory.
template <typename T, int QL>
__global__ void __launch_bounds__(kThreads) selective_step_kernel(T* __restrict__ out, const T* __restrict__ a_log,
                                                                  const T* __restrict__ skip, const T* __restrict__ dt_bias,
                                                                  ScanParams p) {
  pdl_trigger();
  const int lane = threadIdx.x & 31, q = lane % QL, r = blockIdx.y;
  const int c = (int)((blockIdx.x * (unsigned)kThreads + threadIdx.x) / QL), N = p.N;
  const bool live = c < p.channels;
  float4 A = make_float4(0.f, 0.f, 0.f, 0.f);
  if (live) {      // (weights do not depend on the kernels before)
    const T* from = a_log + (size_t)c * N + 4 * q;
    if (4 * q < N) A.x = -expf(to_f32(from[0]));
    if (4 * q + 1 < N) A.y = -expf(to_f32(from[1]));
    if (4 * q + 2 < N) A.z = -expf(to_f32(from[2]));
    if (4 * q + 3 < N) A.w = -expf(to_f32(from[3]));
  }
  const float bias = live ? to_f32(dt_bias[c]) : 0.f, D = live ? to_f32(skip[c]) : 0.f;
  pdl_wait();
  const int t = p.q_start[r], slot = p.state_slot[r];
  if (p.q_start[r + 1] == t) return;
  if (slot == -1) {       // a row of padding leaves zeros
    if (live && q == 0) out[(size_t)t * p.ld_out + c] = from_f32<T>(0.f);
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (threadIdx.x == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  float4 S = make_float4(0.f, 0.f, 0.f, 0.f), b = S, cc = S;
  float* st = p.state + ((size_t)slot * p.channels + (live ? c : 0)) * N + 4 * q;
  const float *row_b = p.bc + (size_t)t * p.ld_bc + p.b_at + 4 * q, *row_c = p.bc + (size_t)t * p.ld_bc + p.c_at + 4 * q;
  auto four = [&](float4& v, const float* from) {
    if (4 * q < N) v.x = from[0];
    if (4 * q + 1 < N) v.y = from[1];
    if (4 * q + 2 < N) v.z = from[2];
    if (4 * q + 3 < N) v.w = from[3];
  };
  if (live && (p.vec & VEC_STATE)) {
    if (4 * q < N) S = load4(st);
  } else if (live) {
    four(S, st);
  }
  if (p.vec & VEC_BC) {
    if (4 * q < N) b = load4(row_b), cc = load4(row_c);
  } else {
    four(b, row_b), four(cc, row_c);
  }
  const float x = live ? p.x[(size_t)t * p.ld_x + c] : 0.f, z = live ? p.z[(size_t)t * p.ld_z + c] : 0.f;
  const float dt = live ? softplus_f(p.dt_pre[(size_t)t * p.ld_dt + c] + bias) : 0.f, dx = dt * x;
  auto step = [&](float& s, float a, float bb, float c4, int e) {
    s = fmaf(expf(dt * a), s, dx * bb);
    if (4 * q + e >= N) s = 0.f;
    return 4 * q + e < N ? s * c4 : 0.f;
  };
  const float4 part = make_float4(step(S.x, A.x, b.x, cc.x, 0), step(S.y, A.y, b.y, cc.y, 1), step(S.z, A.z, b.z, cc.z, 2),
                                  step(S.w, A.w, b.w, cc.w, 3));
  float4 sum;
#pragma unroll
  for (int i = 0; i < QL; ++i) {
    const int from = lane - q + i;
    const float px = __shfl_sync(0xffffffffu, part.x, from), py = __shfl_sync(0xffffffffu, part.y, from);
    const float pz = __shfl_sync(0xffffffffu, part.z, from), pw = __shfl_sync(0xffffffffu, part.w, from);
    if (i == 0) sum = make_float4(px, py, pz, pw);
    else sum.x += px, sum.y += py, sum.z += pz, sum.w += pw;
  }
  if (!live) return;
  if (q == 0) out[(size_t)t * p.ld_out + c] = from_f32<T>(fmaf(D, x, (sum.x + sum.z) + (sum.y + sum.w)) * silu_f(z));
  if (!p.write) return;
  if (p.vec & VEC_STATE) {
    if (4 * q < N) store4(st, S);
    return;
  }
  if (4 * q < N) st[0] = S.x;
  if (4 * q + 1 < N) st[1] = S.y;
  if (4 * q + 2 < N) st[2] = S.z;
  if (4 * q + 3 < N) st[3] = S.w;
}

template <typename T, int LN, int WARPS, int WTS>
int launch_walk_as(void* out, const void* a_log, const void* skip, const void* dt_bias, const ScanParams& p, int requests,
                   cudaStream_t stream) {
  constexpr int WC = WARPS * (32 / LN);
  const long long ctas = (long long)((p.channels + WC - 1) / WC) * requests, sms = lab_sm_count();
  size_t smem = sizeof(float) * ScanTile(WC, LN, WTS, WARPS).total;
  // A long walk of few CTAs: no more of them a multiprocessor than need be, wherever the kernel before leaves room first
  // (2,048 tokens by 1,792 channels of 16, with the mixer around it, 214 us; 331 where five may settle on one).
  if (WTS == 32 && ctas <= 3 * sms) {
    const size_t each = (size_t)(226 * 1024) / (size_t)((ctas + sms - 1) / sms) - 1024;
    if (each > smem) smem = each / 128 * 128;
  }
  const bool whole = p.N == LN;
  const auto kernel = whole ? selective_walk_kernel<T, LN, WARPS, WTS, true> : selective_walk_kernel<T, LN, WARPS, WTS, false>;
  static LabShared granted[2];
  const cudaError_t e = lab_allow_shared(granted[whole], (const void*)kernel, smem);
  if (e != cudaSuccess) return (int)e;
  return (int)lab_launch(kernel, dim3((p.channels + WC - 1) / WC, requests), dim3(32 * WARPS), smem, stream, (T*)out,
                         (const T*)a_log, (const T*)skip, (const T*)dt_bias, p);
}

template <typename T, int LN>
int launch_walk(void* out, const void* a_log, const void* skip, const void* dt_bias, const ScanParams& p, int requests,
                int longest, cudaStream_t stream) {
  if (longest == 1)
    return (int)lab_launch(selective_step_kernel<T, LN / 4>, dim3((p.channels * (LN / 4) + kThreads - 1) / kThreads, requests),
                           dim3(kThreads), 0, stream, (T*)out, (const T*)a_log, (const T*)skip, (const T*)dt_bias, p);
  if (longest <= 8) return launch_walk_as<T, LN, 8, 8>(out, a_log, skip, dt_bias, p, requests, stream);
  return launch_walk_as<T, LN, 4, 32>(out, a_log, skip, dt_bias, p, requests, stream);
}

template <typename T, int WL, int R, int MODE, bool QUADS>
int launch_scan_as(void* out, const void* a_log, const void* skip, const void* dt_bias, const ScanParams& p, int requests,
                   cudaStream_t stream) {
  constexpr int WC = WTHREADS / WL;
  const size_t smem = sizeof(float) * ((size_t)2 * scan_chunk_floats(WC, (p.N + 3) & ~3) + WT * WC + WT * WTHREADS);
  static LabShared granted;
  const cudaError_t e = lab_allow_shared(granted, (const void*)selective_scan_kernel<T, WL, R, MODE, QUADS>, smem);
  if (e != cudaSuccess) return (int)e;
  const int segments = MODE == SCAN_WHOLE ? 1 : MODE == SCAN_CLOSE ? p.segments - 1 : p.segments;
  return (int)lab_launch(selective_scan_kernel<T, WL, R, MODE, QUADS>, dim3((p.channels + WC - 1) / WC, requests, segments),
                         dim3(WTHREADS), smem, stream, (T*)out, (const T*)a_log, (const T*)skip, (const T*)dt_bias, p);
}

template <typename T, int WL, int R, bool QUADS = true>
int launch_scan(void* out, const void* a_log, const void* skip, const void* dt_bias, const ScanParams& p, int requests,
                cudaStream_t stream) {
  if constexpr (R > 4) {      // (smaller states in one piece have a walk of their own)
    if (p.segments <= 1) return launch_scan_as<T, WL, R, SCAN_WHOLE, QUADS>(out, a_log, skip, dt_bias, p, requests, stream);
  }
  const int e = launch_scan_as<T, WL, R, SCAN_CLOSE, QUADS>(out, a_log, skip, dt_bias, p, requests, stream);
  return e != 0 ? e : launch_scan_as<T, WL, R, SCAN_OUTPUT, QUADS>(out, a_log, skip, dt_bias, p, requests, stream);
}

// Four lanes a channel up to 64 entries; eight beyond, where a lane's registers would not hold a quarter.
template <typename T>
int pick_scan(void* out, const void* a_log, const void* skip, const void* dt_bias, const ScanParams& p, int requests,
              int longest, cudaStream_t stream) {
  if (p.N <= SMALL_STATE && p.segments > 1)
    return p.N % 4 != 0 ? launch_scan<T, 4, 4, false>(out, a_log, skip, dt_bias, p, requests, stream)
                        : launch_scan<T, 4, 4>(out, a_log, skip, dt_bias, p, requests, stream);
  if (p.N <= 4) return launch_walk<T, 4>(out, a_log, skip, dt_bias, p, requests, longest, stream);
  if (p.N <= 8) return launch_walk<T, 8>(out, a_log, skip, dt_bias, p, requests, longest, stream);
  if (p.N <= SMALL_STATE) return launch_walk<T, 16>(out, a_log, skip, dt_bias, p, requests, longest, stream);
  if (p.N % 4 != 0) {
    if (p.N <= 64) return launch_scan<T, 4, 16, false>(out, a_log, skip, dt_bias, p, requests, stream);
    if (p.N <= SCAN_MAX_STATE) return launch_scan<T, 8, 32, false>(out, a_log, skip, dt_bias, p, requests, stream);
    return (int)cudaErrorInvalidValue;
  }
  if (p.N <= 32) return launch_scan<T, 4, 8>(out, a_log, skip, dt_bias, p, requests, stream);
  if (p.N <= 64) return launch_scan<T, 4, 16>(out, a_log, skip, dt_bias, p, requests, stream);
  if (p.N <= 128) return launch_scan<T, 8, 16>(out, a_log, skip, dt_bias, p, requests, stream);
  if (p.N <= SCAN_MAX_STATE) return launch_scan<T, 8, 32>(out, a_log, skip, dt_bias, p, requests, stream);
  return (int)cudaErrorInvalidValue;
}
}  // namespace

// The largest state (entries per channel) the walk takes.
LAB_EXPORT int lab_selective_scan_max_state() { return SCAN_MAX_STATE; }

LAB_EXPORT int lab_conv_silu(float* out32, void* out_t, const float* proj, int ld, int conv_at, int channels, int taps,
                             const void* taps_w, const void* taps_b, float* kept, const int* row_req,
                             const int* q_start, const int* state_slot, int tokens, int requests, int n_slots,
                             int write, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (taps < 1 || channels <= 0) return (int)cudaErrorInvalidValue;
  ConvParams p;
  p.proj = proj; p.ld = ld; p.conv_at = conv_at; p.channels = channels; p.taps = taps; p.kept = kept;
  p.row_req = row_req; p.q_start = q_start; p.state_slot = state_slot; p.n_slots = n_slots;
  const int c_blocks = (channels + kThreads - 1) / kThreads;
  if (c_blocks > 65535) return (int)cudaErrorInvalidValue;
  cudaError_t e;
  // few rows: a thread a row, so that all of them are read at once (300 x 1,792: 5.1 us, 7.1 by eights)
  const bool many = taps == 4 && (long long)tokens * channels >= 1500000;
  const dim3 tiles((tokens + CONV_ROWS - 1) / CONV_ROWS, c_blocks);
  if (many && dtype == LAB_F32)
    e = lab_launch(conv_silu4_kernel<float>, tiles, dim3(kThreads), 0, stream, out32, (float*)nullptr, (const float*)taps_w,
                   (const float*)taps_b, p, tokens);
  else if (many)
    e = lab_launch(conv_silu4_kernel<__nv_bfloat16>, tiles, dim3(kThreads), 0, stream, out32, (__nv_bfloat16*)out_t,
                   (const __nv_bfloat16*)taps_w, (const __nv_bfloat16*)taps_b, p, tokens);
  else if (dtype == LAB_F32)
    e = lab_launch(conv_silu_kernel<float>, dim3(tokens, c_blocks), dim3(kThreads), 0, stream, out32, (float*)nullptr,
                   (const float*)taps_w, (const float*)taps_b, p);
  else
    e = lab_launch(conv_silu_kernel<__nv_bfloat16>, dim3(tokens, c_blocks), dim3(kThreads), 0, stream, out32,
                   (__nv_bfloat16*)out_t, (const __nv_bfloat16*)taps_w, (const __nv_bfloat16*)taps_b, p);
  if (e != cudaSuccess) return (int)e;
  if (write && taps > 1)
    return (int)lab_launch(conv_keep_inputs_kernel, dim3(requests, c_blocks), dim3(kThreads), 0, stream, p);
  return 0;
}

// segments > 1: every request's rows are cut into at most that many; `states` [requests, segments, channels, N] and
// `sums` [requests, segments, channels] are scratch.
LAB_EXPORT int lab_selective_scan(void* out, int ld_out, const float* x, int ld_x, const float* dt_pre, int ld_dt,
                                  const float* bc, int ld_bc, int b_at, int c_at, const float* z, int ld_z,
                                  const void* a_log, const void* skip, const void* dt_bias, float* state,
                                  const int* q_start, const int* state_slot, int requests, int channels, int N,
                                  int n_slots, int write, int longest, int segments, float* states, float* sums,
                                  int dtype, cudaStream_t stream) {
  if (requests <= 0) return 0;
  if (channels <= 0 || N <= 0 || N > SCAN_MAX_STATE) return (int)cudaErrorInvalidValue;
  if (segments > 65535 || (segments > 1 && (states == nullptr || sums == nullptr))) return (int)cudaErrorInvalidValue;
  ScanParams p;
  p.x = x; p.dt_pre = dt_pre; p.bc = bc; p.z = z; p.state = state; p.q_start = q_start; p.state_slot = state_slot;
  p.ld_x = ld_x; p.ld_dt = ld_dt; p.ld_bc = ld_bc; p.ld_z = ld_z; p.b_at = b_at; p.c_at = c_at; p.channels = channels;
  p.N = N; p.n_slots = n_slots; p.write = write; p.ld_out = ld_out;
  p.segments = segments; p.states = states; p.sums = sums;
  const int unit = dtype == LAB_F32 ? 4 : 8;
  auto on_16 = [](const void* a) { return ((uintptr_t)a & 15) == 0; };
  const bool rows = ((ld_x | ld_dt | ld_z | channels) & 3) == 0 && on_16(x) && on_16(dt_pre) && on_16(z);
  const bool both = ((ld_bc | b_at | c_at | N) & 3) == 0 && on_16(bc);
  p.vec = N > SMALL_STATE || segments > 1 ? rows && both
                                          : rows * VEC_ROWS + both * VEC_BC + (N % 4 == 0 && on_16(state)) * VEC_STATE +
                                                (channels % unit == 0 && ld_out % unit == 0 && on_16(out)) * VEC_OUT;
  if (requests > 65535) return (int)cudaErrorInvalidValue;
  if (dtype == LAB_F32) return pick_scan<float>(out, a_log, skip, dt_bias, p, requests, longest, stream);
  return pick_scan<__nv_bfloat16>(out, a_log, skip, dt_bias, p, requests, longest, stream);
}
