// Recurrent mixers whose state per head is a matrix S [key channel, value channel] with a scalar decay:
//
//     S_t = a_t * S_{t-1} + (s_t * k_t) v_t^T,        o_t = S_t^T q_t
//
// a_t is a constant of the head (linear attention with a fixed decay) or a number per token and head (a
// state-space mixer, where a_t = exp(-exp(A_log) * dt_t) and s_t = dt_t); q and k may be shared by the
// heads of a group.  The state is 32-bit, is read at a request's first row of the step and written back
// after its last, and every product and sum of the recurrence is 32-bit.
//
//   decay_scan        the recurrence over each request's rows (any number of rows, single tokens included), token by
//                     token in order; rows of a long portion in segments side by side, whose opening states follow
//                     from the segments before them (S <- (product of decays) S + S_segment)
//   ssm_prepare       for a state-space mixer, from the 32-bit input projection [z | x | B | C | dt]: the
//                     causal convolution per channel of x, B, C over the last `taps` inputs (the inputs
//                     before a step's first row come from the request's kept inputs) with bias and SiLU;
//                     dt = softplus(dt + dt_bias); a = exp(-exp(A_log) * dt)
//   ssm_keep_inputs   the request's last taps - 1 inputs of x, B, C replace the kept ones
//   gated_norm        the heads' outputs side by side (+ skip * x), a gate, an RMS norm in equal parts with
//                     a weight, in either order (gate first with SiLU, or norm first with a sigmoid),
//                     rounded to T for the output projection
//
// T says how weights are stored and how the last result is rounded.
#include "chunks.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int SCAN_P = 4;     // threads that share one column of the state
constexpr int SCAN_CT = 16;   // tokens staged per chunk
constexpr int LONG_WALK = 256;      // tokens from which the next kernel is let in at the walk's end only

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float sigmoid_f(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct ScanParams {
  float* out;            // [tokens, ld_o]: head h at h * V
  int ld_o;
  const float* q;        // [tokens, ld_qk]: group g at g * N
  const float* k;
  int ld_qk;
  const float* v;        // [tokens, ld_v]: head h at h * V
  int ld_v;
  const float* a_tok;    // [tokens, ld_a] decay per token and head, or null
  const float* s_tok;    // [tokens, ld_a] scale of the key per token and head, or null (1)
  int ld_a;
  const float* a_head;   // [H] decay per head, read when a_tok is null
  float* state;          // [slots, H, N, V]
  const int* q_start;
  const int* state_slot;
  int n_slots, H, G, N, V, act, write;
  int vec;               // q, k, v rows may be copied 16 bytes at a time
  int segments;          // a request's rows are cut into at most that many segments of whole chunks
  float* states;         // [requests, segments, H, N, V]: 0, a copy of the request's state; i, the state at the end of
                         // segment i - 1 (from zeros, of segment 0 from the request's state)
  float* decays;         // [requests, segments, H]: the product of the decays of segment i - 1
};
// What a launch does: everything in one piece, the segments' closing states, or the outputs.
enum { SCAN_WHOLE, SCAN_CLOSE, SCAN_OUTPUT };


// grid (slices of V, heads, requests); block 2 * SCAN_P * Vs threads in two halves.
//
// Walkers (the first SCAN_P * Vs threads): thread (j, part) keeps rows part * R .. part * R + R - 1 of column
// slice * Vs + j of the state in registers (R a multiple of 4: the rows' keys and queries come from shared
// memory four at a time; the four threads' shares of a token's keys lie R + 4 floats apart, which spreads
// their 16-byte loads over the banks).  A token costs a walker 3 R / 2 instructions on two rows each behind R / 2 loads;
// the four walkers of a column add their shares of four tokens' outputs by three shuffles together.
// The walk of a segment is one dependent chain: its time is the number of tokens times that step, whatever the number
// of CTAs, so nothing else may sit on it.  (A launch for the closing states forms no outputs: no queries, two thirds
// of the instructions.)
//
// Helpers (the other half) keep everything else off that chain: while the walkers are on chunk c (16 tokens),
// the helpers apply the SiLU to chunk c + 1, whose rows their cp.async copies have brought (16 bytes a copy
// where the operands' addresses allow it: `vec`), and start the copies of chunk c + 2 into the buffer the
// walkers left one chunk ago.  Three buffers, one barrier of the whole CTA per chunk.
template <int R, int MODE>
__device__ __forceinline__ void decay_scan(const ScanParams& p) {
  extern __shared__ __align__(16) float smem[];
  constexpr int RS = R + 4;                      // floats between two threads' shares of a token's keys
  constexpr int NP = SCAN_P * RS;                // floats of a token's keys (or queries) in shared memory
  constexpr bool OUT = MODE != SCAN_CLOSE;
  const int walkers = blockDim.x / 2, Vs = walkers / SCAN_P;
  const int tok_floats = 2 * NP + Vs + 4;        // k | q | v | a | s | (two unused, which keep rows 16-byte aligned)
  const int segments = MODE == SCAN_WHOLE ? 1 : MODE == SCAN_CLOSE ? p.segments - 1 : p.segments;
  const int h = blockIdx.y, r = blockIdx.z / segments, seg = blockIdx.z % segments, g = h / (p.H / p.G);
  const bool helper = threadIdx.x >= walkers;
  const int tid = helper ? threadIdx.x - walkers : threadIdx.x;      // index within the half
  const int j = tid / SCAN_P, part = tid % SCAN_P;
  const int col0 = blockIdx.x * Vs, col = col0 + j;
  int t0 = p.q_start[r], n_tok = p.q_start[r + 1] - t0, last = 0;      // last: the request's last segment
  const int slot = p.state_slot[r];
  if (MODE != SCAN_WHOLE && n_tok > 0) {
    const int len = ((n_tok + p.segments - 1) / p.segments + SCAN_CT - 1) / SCAN_CT * SCAN_CT;
    last = (n_tok - 1) / len;
    t0 += seg * len;
    n_tok = MODE == SCAN_CLOSE && seg >= last ? 0 : min(len, n_tok - seg * len);
  }
  if (MODE == SCAN_WHOLE && n_tok < LONG_WALK) pdl_trigger();
  if (n_tok <= 0 || slot == -1) {      // nothing to do, or rows of padding (their output is never read)
    pdl_wait();
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (threadIdx.x == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    pdl_wait();
    return;
  }
  // padding of the key channels and of the columns stays zero for the whole walk: the copies never touch it
  for (int i = threadIdx.x; i < 3 * SCAN_CT * tok_floats; i += blockDim.x) smem[i] = 0.f;
  __syncthreads();
  pdl_wait();

  const int n_chunks = (n_tok + SCAN_CT - 1) / SCAN_CT;
  const int v_cols = min(Vs, p.V - col0);
  auto buffer = [&](int chunk) { return smem + (chunk % 3) * SCAN_CT * tok_floats; };

  // ---- helpers' pieces ----
  auto at = [](int n) { return (n / R) * RS + (n % R); };      // where key channel n lies within a token's keys
  // One loop over all of a chunk's copies (tokens x pieces), so that every helper has a few copies in flight
  // instead of the helpers walking the tokens one after the other.
  auto issue = [&](int chunk) {
    const int first = chunk * SCAN_CT, cnt = min(SCAN_CT, n_tok - first);
    float* base = buffer(chunk);
    const float* k0 = p.k + (size_t)(t0 + first) * p.ld_qk + g * p.N;
    const float* q0 = p.q + (size_t)(t0 + first) * p.ld_qk + g * p.N;
    const float* v0 = p.v + (size_t)(t0 + first) * p.ld_v + h * p.V + col0;
    if (p.vec) {
      const int nk = p.N / 4, nv = v_cols / 4, per = 2 * nk + nv;
      for (int e = tid; e < cnt * per; e += walkers) {
        const int tt = e / per, c = e - tt * per;
        float* dst = base + tt * tok_floats;
        if (c < nk) cp_async16(dst + at(4 * c), k0 + (size_t)tt * p.ld_qk + 4 * c);
        else if (c < 2 * nk) { if (OUT) cp_async16(dst + NP + at(4 * (c - nk)), q0 + (size_t)tt * p.ld_qk + 4 * (c - nk)); }
        else cp_async16(dst + 2 * NP + 4 * (c - 2 * nk), v0 + (size_t)tt * p.ld_v + 4 * (c - 2 * nk));
      }
    } else {
      const int per = 2 * p.N + v_cols;
      for (int e = tid; e < cnt * per; e += walkers) {
        const int tt = e / per, c = e - tt * per;
        float* dst = base + tt * tok_floats;
        if (c < p.N) cp_async4(dst + at(c), k0 + (size_t)tt * p.ld_qk + c);
        else if (c < 2 * p.N) { if (OUT) cp_async4(dst + NP + at(c - p.N), q0 + (size_t)tt * p.ld_qk + (c - p.N)); }
        else cp_async4(dst + 2 * NP + (c - 2 * p.N), v0 + (size_t)tt * p.ld_v + (c - 2 * p.N));
      }
    }
    if (p.a_tok != nullptr && tid < 2 * cnt) {      // a token's decay and key scale: one helper each
      const int tt = tid >> 1, which = tid & 1;
      const float* src = which == 0 ? p.a_tok : p.s_tok;
      if (src != nullptr)
        cp_async4(base + tt * tok_floats + 2 * NP + Vs + which, src + (size_t)(t0 + first + tt) * p.ld_a + h);
    }
  };
  // after the copies of `chunk` have landed for every helper: SiLU of q, k and v, once per element
  auto finish = [&](int chunk) {
    asm volatile("bar.sync 1, %0;" ::"r"(walkers) : "memory");      // the helpers alone
    if (!p.act) return;
    const int cnt = min(SCAN_CT, n_tok - chunk * SCAN_CT), per = (2 * NP + Vs) / 4;
    float* base = buffer(chunk);
    for (int e = tid; e < cnt * per; e += walkers) {
      const int tt = e / per, c = e - tt * per;
      float4* at4 = reinterpret_cast<float4*>(base + tt * tok_floats) + c;
      float4 z = *at4;
      z.x = silu_quick(z.x), z.y = silu_quick(z.y), z.z = silu_quick(z.z), z.w = silu_quick(z.w);
      *at4 = z;
    }
  };

  f32x2 S[R / 2];
  float decayed = 1.f;      // SCAN_CLOSE: the product of the decays
  float* st = p.state + ((size_t)slot * p.H + h) * p.N * p.V;
  const size_t per_segment = (size_t)p.H * p.N * p.V;
  float* kept = MODE == SCAN_WHOLE ? nullptr : p.states + (size_t)r * p.segments * per_segment + (size_t)h * p.N * p.V;
  float* decays = MODE == SCAN_WHOLE ? nullptr : p.decays + (size_t)r * p.segments * p.H + h;
  float a_const = 0.f;
  if (helper) {
    issue(0);
    cp_async_commit_group();
    if (n_chunks > 1) issue(1);
    cp_async_commit_group();
    cp_async_wait_group<1>();
    finish(0);
  } else {
    float s[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const size_t at = (size_t)(part * R + i) * p.V + col;
      s[i] = 0.f;
      if (part * R + i >= p.N || col >= p.V) continue;
      if (MODE == SCAN_WHOLE || (MODE == SCAN_OUTPUT && last == 0)) {
        s[i] = st[at];
      } else if (MODE == SCAN_CLOSE) {
        // (the last segment's CTA of the next launch writes the request's state while others still open theirs)
        if (seg == 0) kept[at] = s[i] = st[at];
      } else {
        s[i] = kept[(seg == 0 ? 0 : per_segment) + at];
      }
    }
    if (MODE == SCAN_OUTPUT) {
      for (int e = 2; e <= seg; ++e) {
        const float a = decays[(size_t)e * p.H];
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (part * R + i < p.N && col < p.V) s[i] = fmaf(a, s[i], kept[e * per_segment + (size_t)(part * R + i) * p.V + col]);
      }
    }
#pragma unroll
    for (int i = 0; i < R / 2; ++i) S[i] = pair_of(s[2 * i], s[2 * i + 1]);
    if (p.a_tok == nullptr) a_const = p.a_head[h];
  }
  __syncthreads();

  for (int c = 0; c < n_chunks; ++c) {
    if (helper) {
      if (c + 2 < n_chunks) issue(c + 2);      // into the buffer the walkers left at the last barrier
      cp_async_commit_group();
      if (c + 1 < n_chunks) {
        cp_async_wait_group<1>();              // all but the copies just started: chunk c + 1 is here
        finish(c + 1);
      }
    } else {
      const int cnt = min(SCAN_CT, n_tok - c * SCAN_CT);
      const float* base = buffer(c);
      float* out = p.out + (size_t)(t0 + c * SCAN_CT) * p.ld_o + h * p.V + col;
      // a token's update; the walker's share of its output
      auto step = [&](int tt) {
        const float* tok = base + tt * tok_floats;
        const ulonglong2* k4 = reinterpret_cast<const ulonglong2*>(tok + part * RS);
        const ulonglong2* q4 = reinterpret_cast<const ulonglong2*>(tok + NP + part * RS);
        const float a = p.a_tok != nullptr ? tok[2 * NP + Vs] : a_const;
        float vj = tok[2 * NP + j];
        if (p.s_tok != nullptr) vj *= tok[2 * NP + Vs + 1];
        const f32x2 aa = pair_of(a, a), vv = pair_of(vj, vj);
        f32x2 acc[2] = {0ull, 0ull};      // zeros
#pragma unroll
        for (int i = 0; i < R / 4; ++i) {
          const ulonglong2 k = k4[i];
          S[2 * i] = fma2(aa, S[2 * i], mul2(k.x, vv));
          S[2 * i + 1] = fma2(aa, S[2 * i + 1], mul2(k.y, vv));
          if (OUT) {
            const ulonglong2 q = q4[i];
            acc[0] = fma2(S[2 * i], q.x, acc[0]);
            acc[1] = fma2(S[2 * i + 1], q.y, acc[1]);
          }
        }
        if (!OUT) decayed *= a;
        return (low_of(acc[0]) + high_of(acc[0])) + (low_of(acc[1]) + high_of(acc[1]));
      };
      // four tokens at a time: their sums over a column's four walkers take three shuffles together and leave walker p
      // with token p's, and the next tokens' arithmetic does not wait for them
      int tt = 0;
      for (; tt + SCAN_P <= cnt; tt += SCAN_P) {
        float t[SCAN_P];
#pragma unroll
        for (int u = 0; u < SCAN_P; ++u) t[u] = step(tt + u);
        if (OUT) {
          const bool hi2 = part & 2, hi1 = part & 1;
          const float s0 = (hi2 ? t[2] : t[0]) + __shfl_xor_sync(0xffffffffu, hi2 ? t[0] : t[2], 2);
          const float s1 = (hi2 ? t[3] : t[1]) + __shfl_xor_sync(0xffffffffu, hi2 ? t[1] : t[3], 2);
          const float total = (hi1 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, hi1 ? s0 : s1, 1);
          if (col < p.V) out[(size_t)(tt + part) * p.ld_o] = total;
        }
      }
      for (; tt < cnt; ++tt) {
        float total = step(tt);
        if (OUT) {
          total += __shfl_xor_sync(0xffffffffu, total, 2);
          total += __shfl_xor_sync(0xffffffffu, total, 1);
          if (part == 0 && col < p.V) out[(size_t)tt * p.ld_o] = total;
        }
      }
    }
    __syncthreads();
  }
  pdl_trigger();      // (not earlier: the next kernel's blocks would settle beside this one's and slow them down)
  if (helper) {
    cp_async_wait_group<0>();
  } else if (MODE == SCAN_CLOSE || (p.write && seg == last)) {
    float* to = MODE == SCAN_CLOSE ? kept + (seg + 1) * per_segment : st;
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int n = part * R + i;
      if (n < p.N && col < p.V) to[(size_t)n * p.V + col] = i % 2 == 0 ? low_of(S[i / 2]) : high_of(S[i / 2]);
    }
    if (MODE == SCAN_CLOSE && blockIdx.x == 0 && tid == 0) decays[(size_t)(seg + 1) * p.H] = decayed;
  }
}

template <int R, int MODE>
__global__ void __launch_bounds__(256) decay_scan_kernel(ScanParams p) {
  decay_scan<R, MODE>(p);
}
// More than 64 key channels in one piece: registers for as many CTAs as shared memory allows, three a multiprocessor up to
// 128 channels, two beyond, for steps that have so many (a long walk of few CTAs is shorter with all the registers it wants).
// Measured, 12 heads of 128 x 128: 64 single tokens 49 us against 55 with two CTAs a multiprocessor, eight requests of 250
// 150 against 168; one of 300 (48 CTAs) 88 with all its registers, 98 without.
template <int R>
__global__ void __launch_bounds__(256, R <= 32 ? 3 : 2) decay_scan_dense_kernel(ScanParams p) {
  decay_scan<R, SCAN_WHOLE>(p);
}

// ---- portions of a prompt: chunks of rows side by side ------------------------------------------
// The recurrence with its sums regrouped into products of small matrices: a first kernel forms every chunk's own contribution
// to the state, a second one runs through a request's chunks and leaves the state before each, a third one forms the outputs
// (chunks.cuh).  A chunk's contribution is sum_j g_63,j s_j k_j v_j^T.  Measured, two requests of 1,000 rows, 14 heads of
// 64 x 68 (us): 15, 5 and 36, against 84 and 36 of the walk's two launches in 7 segments.  The products on the tensor cores as
// sums of two TF32 values (mma.sync) took as long, 14 and 43, with two to three times the error.

// grid (places of chunks, heads, slices of N of 64 x slices of V of Vs): sum_j g_63,j s_j k_j v_j^T in place `at` of
// p.states [places, H, N, V]; the product of the chunk's decays in p.decays [places, H].
template <bool VEC>
__global__ void __launch_bounds__(CHUNK_THREADS) chunk_close_kernel(ScanParams p, int requests, int Vs, int slices) {
  __shared__ __align__(16) float ks[CHUNK * 64], vs[CHUNK * WIDE], weight[CHUNK];
  pdl_wait();
  const int at = blockIdx.x, h = blockIdx.y, g = h / (p.H / p.G), tid = threadIdx.x;
  const int n0 = blockIdx.z / slices * 64, col0 = blockIdx.z % slices * Vs, cols = min(Vs, p.V - col0), keys = min(64, p.N - n0);
  int row0, rows;
  chunk_rows(p.q_start, p.state_slot, requests, p.n_slots, at, row0, rows);
  if (rows == 0) return;
  const int quads = (cols + 3) / 4;
  if (tid < 32) {      // two rows a lane: the product of the decays after each
    float a[2], s[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = 2 * tid + i;
      a[i] = t >= rows ? 1.f : p.a_tok != nullptr ? p.a_tok[(size_t)(row0 + t) * p.ld_a + h] : p.a_head[h];
      s[i] = t >= rows ? 0.f : p.s_tok != nullptr ? p.s_tok[(size_t)(row0 + t) * p.ld_a + h] : 1.f;
    }
    float after = a[0] * a[1];      // of this lane's rows and those behind
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float right = __shfl_down_sync(0xffffffffu, after, o);
      if (tid + o < 32) after *= right;
    }
    const float behind = __shfl_down_sync(0xffffffffu, after, 1), w1 = tid < 31 ? behind : 1.f;
    weight[2 * tid] = a[1] * w1 * s[0], weight[2 * tid + 1] = w1 * s[1];
    if (tid == 0 && blockIdx.z == 0) p.decays[(size_t)at * p.H + h] = after;
  }
  const float4 zeros = make_float4(0.f, 0.f, 0.f, 0.f);
  const Divider by_c(quads);
  copy_quads(CHUNK * 16, [&](int e) {
    return e / 16 < rows ? row4<VEC>(p.k + (size_t)(row0 + e / 16) * p.ld_qk + g * p.N + n0, 4 * (e % 16), keys) : zeros;
  }, [&](int e, float4 z) { store4(ks + 4 * e, act4(z, p.act)); });
  __syncthreads();      // the weights
  copy_quads(CHUNK * quads, [&](int e) {
    return by_c.over(e) < rows ? row4<VEC>(p.v + (size_t)(row0 + by_c.over(e)) * p.ld_v + h * p.V + col0, 4 * by_c.rest(e), cols) : zeros;
  }, [&](int e, float4 z) {
    const float w = weight[by_c.over(e)];
    z = act4(z, p.act);
    store4(vs + by_c.over(e) * WIDE + 4 * by_c.rest(e), make_float4(z.x * w, z.y * w, z.z * w, z.w * w));
  });
  __syncthreads();
  const int n = by_c.over(tid) * 8, c = by_c.rest(tid) * 4;
  if (n >= keys) return;
  Tile acc;
  acc.clear();
  for (int t0 = 0; t0 < CHUNK; t0 += RUN) {
    Tile part;
    part.clear();
#pragma unroll 4
    for (int t = t0; t < t0 + RUN; ++t) part.step(ks + t * 64 + n, ks + t * 64 + n + 4, vs + t * WIDE + c);
    acc.add(part);
  }
  float* dst = p.states + (((size_t)at * p.H + h) * p.N + n0 + n) * p.V + col0 + c;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (n + i >= keys) break;
    if (VEC) store4(dst + (size_t)i * p.V, make_float4(acc.get(i, 0), acc.get(i, 1), acc.get(i, 2), acc.get(i, 3)));
    else
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < cols) dst[(size_t)i * p.V + j] = acc.get(i, j);
  }
}

// grid (blocks of N V entries, heads, requests): an entry of the state a thread, through the request's chunks in order; what a
// chunk contributes makes way for the state before it.
__global__ void __launch_bounds__(256) chunk_open_kernel(ScanParams p) {
  pdl_wait();
  const int h = blockIdx.y, r = blockIdx.z, e = blockIdx.x * 256 + threadIdx.x, first = p.q_start[r], rows = p.q_start[r + 1] - first;
  const int slot = p.state_slot[r], NV = p.N * p.V;
  if (rows <= 0 || slot == -1 || e >= NV) return;
  if (slot < 0 || slot >= p.n_slots) {
    if (e == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  float* state = p.state + ((size_t)slot * p.H + h) * NV + e;
  const int chunks = (rows + CHUNK - 1) / CHUNK;
  const size_t at = (size_t)first_chunk(first, r) * p.H + h, next = p.H;
  float* own = p.states + at * NV + e;
  const float* decay = p.decays + at;
  float S = *state;
  constexpr int AHEAD = 8;
  float l[AHEAD], a[AHEAD];
  for (int c0 = 0; c0 < chunks; c0 += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c0 + i < chunks) l[i] = own[(c0 + i) * next * NV], a[i] = decay[(c0 + i) * next];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i)
      if (c0 + i < chunks) {
        own[(c0 + i) * next * NV] = S;
        S = fmaf(a[i], S, l[i]);
      }
  }
  if (p.write) *state = S;
  pdl_trigger();
}

// ---- state-space mixer: convolution, step sizes, decays ---------------------------------------
struct SsmParams {
  const float* proj;     // [tokens, ld]
  int ld, conv_at, dt_at, channels, taps, H;
  float* kept;           // [slots, taps - 1, channels]: the request's last inputs, oldest first
  const int* row_req;
  const int* q_start;
  const int* state_slot;
  int n_slots;
};

template <typename T>
__global__ void __launch_bounds__(kThreads) ssm_prepare_kernel(float* __restrict__ conv_out, float* __restrict__ dt_out,
                                                               float* __restrict__ a_out, const T* __restrict__ taps_w,
                                                               const T* __restrict__ taps_b, const T* __restrict__ dt_bias,
                                                               const T* __restrict__ a_log, SsmParams p) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, r = p.row_req[t], first = p.q_start[r], slot = p.state_slot[r];
  const int K = p.taps, C = p.channels;
  // grid (rows, blocks of channels): a thread forms one channel, so that a row's loads are all in flight at
  // once (a step of few rows is bound by their latency); the first block of a row also forms its step sizes
  const int c = blockIdx.y * kThreads + threadIdx.x;
  const bool heads_too = blockIdx.y == 0;
  if (slot == -1) {       // a row of padding
    if (c < C) conv_out[(size_t)t * C + c] = 0.f;
    for (int h = threadIdx.x; heads_too && h < p.H; h += kThreads) dt_out[(size_t)t * p.H + h] = a_out[(size_t)t * p.H + h] = 0.f;
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (threadIdx.x == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  const float* kept = p.kept + (size_t)slot * (K - 1) * C;
  if (c < C) {
    float acc = to_f32(taps_b[c]);
    for (int jj = 0; jj < K; ++jj) {
      const int src = t - (K - 1) + jj;       // the last tap meets the row itself
      const float u = src >= first ? p.proj[(size_t)src * p.ld + p.conv_at + c]
                                   : kept[(size_t)((K - 1) + (src - first)) * C + c];
      acc = fmaf(to_f32(taps_w[(size_t)c * K + jj]), u, acc);
    }
    conv_out[(size_t)t * C + c] = silu_f(acc);
  }
  for (int h = threadIdx.x; heads_too && h < p.H; h += kThreads) {
    const float dt = softplus_f(p.proj[(size_t)t * p.ld + p.dt_at + h] + to_f32(dt_bias[h]));
    dt_out[(size_t)t * p.H + h] = dt;
    a_out[(size_t)t * p.H + h] = expf(-expf(to_f32(a_log[h])) * dt);
  }
}

// grid (requests, blocks of channels), after every row of the step has read the kept inputs.  A thread walks
// the kept rows of its one channel oldest first: what it overwrites it has already moved.
__global__ void __launch_bounds__(kThreads) ssm_keep_inputs_kernel(SsmParams p, int requests) {
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

// ---- gate and norm of the heads' outputs ------------------------------------------------------
// y[i] = o[t, i] + skip[head of i] * x[t, i]; gate_first: y *= silu(gate), then y / rms(part of i) * w;
// else y / rms(part) * w * sigmoid(gate); times `mult`, rounded to T.
template <typename T>
__global__ void __launch_bounds__(kThreads) gated_norm_kernel(T* __restrict__ out, int ld_out, const float* __restrict__ o,
                                                              int ld_o, const float* __restrict__ x, int ld_x,
                                                              const T* __restrict__ skip, int head_size,
                                                              const float* __restrict__ gate, int ld_g,
                                                              const T* __restrict__ w, int width, int parts,
                                                              int gate_first, float eps, float mult) {
  extern __shared__ float row[];      // [width]
  __shared__ float scratch[32];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const int part_size = width / parts;
  for (int i = threadIdx.x; i < width; i += kThreads) {
    float y = o[(size_t)t * ld_o + i];
    if (skip != nullptr) y = fmaf(to_f32(skip[i / head_size]), x[(size_t)t * ld_x + i], y);
    if (gate_first) y *= silu_f(gate[(size_t)t * ld_g + i]);
    row[i] = y;
  }
  __syncthreads();
  for (int g = 0; g < parts; ++g) {
    float ss = 0.f;
    for (int i = threadIdx.x; i < part_size; i += kThreads) {
      const float y = row[g * part_size + i];
      ss += y * y;
    }
    ss = block_sum(ss, scratch);
    const float inv = 1.0f / sqrtf(ss / (float)part_size + eps);
    for (int i = threadIdx.x; i < part_size; i += kThreads) {
      const int c = g * part_size + i;
      float y = row[c] * inv * to_f32(w[c]);
      if (!gate_first) y *= sigmoid_f(gate[(size_t)t * ld_g + c]);
      out[(size_t)t * ld_out + c] = from_f32<T>(y * mult);
    }
  }
}

template <int R, int MODE>
int launch_scan_as(const ScanParams& p, int requests, int vs, cudaStream_t stream) {
  const size_t smem = (size_t)3 * SCAN_CT * (2 * SCAN_P * (R + 4) + vs + 4) * sizeof(float);
  const int segments = MODE == SCAN_WHOLE ? 1 : MODE == SCAN_CLOSE ? p.segments - 1 : p.segments;
  const dim3 grid((p.V + vs - 1) / vs, p.H, requests * segments), block(2 * SCAN_P * vs);
  if constexpr (MODE == SCAN_WHOLE && R > 16) {
    if ((long long)grid.x * grid.y * grid.z > (R <= 32 ? 2 : 1) * lab_sm_count()) {
      static LabShared granted;
      const cudaError_t e = lab_allow_shared(granted, (const void*)decay_scan_dense_kernel<R>, smem);
      if (e != cudaSuccess) return (int)e;
      return (int)lab_launch(decay_scan_dense_kernel<R>, grid, block, smem, stream, p);
    }
  }
  static LabShared granted;
  const cudaError_t e = lab_allow_shared(granted, (const void*)decay_scan_kernel<R, MODE>, smem);
  if (e != cudaSuccess) return (int)e;
  return (int)lab_launch(decay_scan_kernel<R, MODE>, grid, block, smem, stream, p);
}

template <int R>
int launch_scan(const ScanParams& p, int requests, int vs, cudaStream_t stream) {
  if (p.segments <= 1) return launch_scan_as<R, SCAN_WHOLE>(p, requests, vs, stream);
  if constexpr (R > 32) {      // (fewer key channels go in chunks)
    const int e = launch_scan_as<R, SCAN_CLOSE>(p, requests, vs, stream);
    return e != 0 ? e : launch_scan_as<R, SCAN_OUTPUT>(p, requests, vs, stream);
  }
  return (int)cudaErrorInvalidValue;
}

// Three launches: see "portions of a prompt".
int launch_chunks(const ScanParams& p, int requests, int tokens, cudaStream_t stream) {
  const int Vs = chunk_slice(p.V), slices = (p.V + Vs - 1) / Vs;
  cudaError_t e = lab_launch(p.vec ? chunk_close_kernel<true> : chunk_close_kernel<false>,
                             dim3(first_chunk(tokens, requests), p.H, (p.N + 63) / 64 * slices), dim3(CHUNK_THREADS), 0, stream, p, requests, Vs, slices);
  if (e != cudaSuccess) return (int)e;
  e = lab_launch(chunk_open_kernel, dim3((p.N * p.V + 255) / 256, p.H, requests), dim3(256), 0, stream, p);
  if (e != cudaSuccess) return (int)e;
  ChunkParams c;
  c.out = p.out; c.ld_o = p.ld_o; c.q = p.q; c.k = p.k; c.ld_qk = p.ld_qk; 
  c.v = p.v; c.ld_v = p.ld_v; c.a = p.a_tok != nullptr ? p.a_tok : p.a_head; c.a_row = p.a_tok != nullptr ? p.ld_a : 0; c.a_head = 1;
  c.s = p.s_tok; c.states = p.states; c.q_start = p.q_start; c.state_slot = p.state_slot; c.requests = requests;
  c.n_slots = p.n_slots; c.H = p.H; c.G = p.G; c.N = p.N; c.V = p.V; c.act = p.act; c.vec = p.vec;
  return launch_chunk_outputs(c, tokens, stream);
}

}  // namespace

// Places of chunks (states of N x V and a decay per place and head) that `lab_decay_scan` wants for a step in chunks.
LAB_EXPORT int lab_decay_scan_places(int tokens, int requests) { return first_chunk(tokens, requests); }

// Largest key size the recurrence kernel is built for.
LAB_EXPORT int lab_decay_scan_max_keys() { return SCAN_P * 64; }

// vs: columns of the state a CTA takes (8, 16 or 32).  segments > 1: every request's rows are cut into at most that many;
// `states` [requests, segments, H, N, V] and `decays` [requests, segments, H] are scratch.  chunk_tokens > 0 (up to 128 key
// channels): the step's rows, which are taken in chunks side by side; the scratch is then [places, H, N, V] and [places, H].
LAB_EXPORT int lab_decay_scan(float* out, int ld_o, const float* q, const float* k, int ld_qk, const float* v, int ld_v,
                              const float* a_tok, const float* s_tok, int ld_a, const float* a_head, float* state,
                              const int* q_start, const int* state_slot, int requests, int n_slots, int H, int G, int N,
                              int V, int act, int write, int vs, int segments, int chunk_tokens, float* states,
                              float* decays, cudaStream_t stream) {
  if (requests <= 0) return 0;
  if (segments > 1 && (states == nullptr || decays == nullptr || (long long)requests * segments > 65535))
    return (int)cudaErrorInvalidValue;
  if (H <= 0 || G <= 0 || H % G || N <= 0 || V <= 0 || (vs != 8 && vs != 16 && vs != 32)) return (int)cudaErrorInvalidValue;
  if (a_tok == nullptr && a_head == nullptr) return (int)cudaErrorInvalidValue;
  ScanParams p;
  p.out = out; p.ld_o = ld_o; p.q = q; p.k = k; p.ld_qk = ld_qk; p.v = v; p.ld_v = ld_v; p.a_tok = a_tok;
  p.s_tok = s_tok; p.ld_a = ld_a; p.a_head = a_head; p.state = state; p.q_start = q_start; p.state_slot = state_slot;
  p.n_slots = n_slots; p.H = H; p.G = G; p.N = N; p.V = V; p.act = act; p.write = write;
  p.segments = segments; p.states = states; p.decays = decays;
  // 16-byte copies: every row of q, k and v, and every head's and slice's start in it, on a 16-byte boundary
  p.vec = N % 4 == 0 && V % 4 == 0 && ld_qk % 4 == 0 && ld_v % 4 == 0 &&
          ((((uintptr_t)q) | ((uintptr_t)k) | ((uintptr_t)v)) & 15) == 0;
  if (chunk_tokens > 0) {
    if (states == nullptr || decays == nullptr || N > 128 || requests > 65535 || H > 65535) return (int)cudaErrorInvalidValue;
    return launch_chunks(p, requests, chunk_tokens, stream);
  }
  if (N <= SCAN_P * 4) return launch_scan<4>(p, requests, vs, stream);
  if (N <= SCAN_P * 8) return launch_scan<8>(p, requests, vs, stream);
  if (N <= SCAN_P * 16) return launch_scan<16>(p, requests, vs, stream);
  if (N <= SCAN_P * 32) return launch_scan<32>(p, requests, vs, stream);
  if (N <= SCAN_P * 64) return launch_scan<64>(p, requests, vs, stream);
  return (int)cudaErrorInvalidValue;
}

LAB_EXPORT int lab_ssm_prepare(float* conv_out, float* dt_out, float* a_out, const float* proj, int ld, int conv_at,
                               int dt_at, int channels, int taps, int H, const void* taps_w, const void* taps_b,
                               const void* dt_bias, const void* a_log, float* kept, const int* row_req,
                               const int* q_start, const int* state_slot, int tokens, int requests, int n_slots,
                               int write, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (taps < 1 || channels <= 0 || H <= 0) return (int)cudaErrorInvalidValue;
  SsmParams p;
  p.proj = proj; p.ld = ld; p.conv_at = conv_at; p.dt_at = dt_at; p.channels = channels; p.taps = taps; p.H = H;
  p.kept = kept; p.row_req = row_req; p.q_start = q_start; p.state_slot = state_slot; p.n_slots = n_slots;
  const int c_blocks = (channels + kThreads - 1) / kThreads;
  if (c_blocks > 65535) return (int)cudaErrorInvalidValue;
  cudaError_t e;
  if (dtype == LAB_F32)
    e = lab_launch(ssm_prepare_kernel<float>, dim3(tokens, c_blocks), dim3(kThreads), 0, stream, conv_out, dt_out, a_out,
                   (const float*)taps_w, (const float*)taps_b, (const float*)dt_bias, (const float*)a_log, p);
  else
    e = lab_launch(ssm_prepare_kernel<__nv_bfloat16>, dim3(tokens, c_blocks), dim3(kThreads), 0, stream, conv_out, dt_out, a_out,
                   (const __nv_bfloat16*)taps_w, (const __nv_bfloat16*)taps_b, (const __nv_bfloat16*)dt_bias,
                   (const __nv_bfloat16*)a_log, p);
  if (e != cudaSuccess) return (int)e;
  if (write && taps > 1)
    return (int)lab_launch(ssm_keep_inputs_kernel, dim3(requests, c_blocks), dim3(kThreads), 0, stream, p, requests);
  return 0;
}

LAB_EXPORT int lab_gated_norm(void* out, int ld_out, const float* o, int ld_o, const float* x, int ld_x, const void* skip,
                              int head_size, const float* gate, int ld_g, const void* w, int tokens, int width, int parts,
                              int gate_first, float eps, float mult, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (parts <= 0 || width % parts) return (int)cudaErrorInvalidValue;
  const size_t smem = (size_t)width * sizeof(float);
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  if (dtype == LAB_F32) {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(gated_norm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    lab_launch(gated_norm_kernel<float>, dim3(tokens), dim3(kThreads), smem, stream, (float*)out, ld_out, o, ld_o, x, ld_x,
               (const float*)skip, head_size, gate, ld_g, (const float*)w, width, parts, gate_first, eps, mult);
  } else {
    if (smem > 48 * 1024)
      cudaFuncSetAttribute(gated_norm_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    lab_launch(gated_norm_kernel<__nv_bfloat16>, dim3(tokens), dim3(kThreads), smem, stream, (__nv_bfloat16*)out, ld_out, o,
               ld_o, x, ld_x, (const __nv_bfloat16*)skip, head_size, gate, ld_g, (const __nv_bfloat16*)w, width, parts,
               gate_first, eps, mult);
  }
  LAB_LAUNCH_CHECK();
}
