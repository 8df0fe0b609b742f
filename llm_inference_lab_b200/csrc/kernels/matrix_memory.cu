// A matrix memory with exponential gates (the mLSTM cell), around the framework's recurrence kernel.
// Per head, with log input gate i_t, log forget gate f_t and a running maximum m (m_0 = 0):
//
//     m_t = max(f_t + m_{t-1}, i_t)
//     S_t = exp(f_t + m_{t-1} - m_t) S_{t-1} + exp(i_t - m_t) k_t v_t^T          S [keys, values]
//     n_t = exp(f_t + m_{t-1} - m_t) n_{t-1} + exp(i_t - m_t) k_t
//     o_t = S_t^T q_t / (max(|n_t . q_t|, exp(-m_t)) + floor)
//
// n rides along as one more column of S: the values get a column of ones (and zeros up to `vpad` columns a
// head, which keeps rows 16-byte aligned), so the recurrence S <- a S + (s k) v^T, o = S^T q of
// `decay_scan` forms S^T q and n . q together.  Here:
//
//   memory_gates      per row, parallel: i = cap tanh((z_i + b_i) / cap), f = logsigmoid(cap tanh((z_f + b_f) / cap));
//                     the values copied with their column of ones
//   memory_stabilize  per request and head, over the step's rows in order: m, the decay a_t and the key scale
//                     s_t of every row; m of the request's last row goes back to its state slot
//   memory_finish     per row: o_t with q's scale, each head over its root mean square, the weight, the sigmoid
//                     gate, rounded to T for the output projection; zeros for rows of padding (state slot -1)
//
// All of it is 32-bit; T says how the weights are stored and how the last result is rounded.
#include "common.cuh"

namespace {
constexpr int kThreads = 256;
// Rows of a request from which the recurrence is let in at the running maximum's end only: its few, long blocks would settle
// beside other kernels' (mixer from a graph, two rows of the state an instruction: 300 tokens 123 us, 84 so; 130 tokens 71, 53).
constexpr int LONG_WALK = 128;

__device__ __forceinline__ float log_sigmoid_f(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

struct GateParams {
  const float* proj;      // [tokens, ld]
  int ld, v_at, i_at, f_at;
  int H, V, vpad;
  float cap;
};

template <typename T>
__global__ void __launch_bounds__(kThreads) memory_gates_kernel(float* __restrict__ gates, float* __restrict__ v_out,
                                                                const T* __restrict__ b_i, const T* __restrict__ b_f,
                                                                GateParams p) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x;
  const float* row = p.proj + (size_t)t * p.ld;
  for (int h = threadIdx.x; h < p.H; h += kThreads) {
    const float zi = row[p.i_at + h] + to_f32(b_i[h]), zf = row[p.f_at + h] + to_f32(b_f[h]);
    gates[((size_t)t * 2) * p.H + h] = p.cap * tanhf(zi / p.cap);
    gates[((size_t)t * 2 + 1) * p.H + h] = log_sigmoid_f(p.cap * tanhf(zf / p.cap));
  }
  const int W = p.H * p.vpad;
  for (int i = threadIdx.x; i < W; i += kThreads) {
    const int h = i / p.vpad, e = i - h * p.vpad;
    v_out[(size_t)t * W + i] = e < p.V ? row[p.v_at + h * p.V + e] : (e == p.V ? 1.f : 0.f);
  }
}

// One warp per (request, head) takes the request's rows 256 at a time, eight neighbouring ones a lane.  Rows f, i take m
// to max(f + m, i), and so do several rows together, with the sum of their f and an i of their own: every lane forms
// that of its rows, a scan over the lanes gives each lane the m before its rows, and it walks them, forming each row's
// two exponentials.  What bounds it is latency (a chain through every row, 32 rows a step, took 51 us for 2,048 rows),
// so the next 256 rows' gates are loaded before this step's arithmetic.  Any m near the running maximum gives the same
// result: both exponentials and the floor of the denominator go by the m that is kept, a lane's first decay by the one
// that the lane before it ends with (the scan's m before its rows may differ from that by roundings).
// in_order: the chain itself, a lane's rows after the other's, so that a row's m does not depend on how the sequence was
// cut into steps; 2,048 rows take about 12 us longer.
// decay[t, h] and scale[t, h] leave as rows of [tokens, 2, H] (over the gates).
__global__ void __launch_bounds__(kThreads) memory_stabilize_kernel(float* __restrict__ gates, float* __restrict__ m_out,
                                                                    float* __restrict__ m_state,
                                                                    const int* __restrict__ q_start,
                                                                    const int* __restrict__ state_slot, int requests,
                                                                    int n_slots, int H, int write, int in_order) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pair = blockIdx.x * (blockDim.x / 32) + warp;
  if (pair >= requests * H) return;
  const int r = pair / H, h = pair - r * H;
  const int t0 = q_start[r], n = q_start[r + 1] - t0, slot = state_slot[r];
  if (n < LONG_WALK) pdl_trigger();
  pdl_wait();
  if (n <= 0 || slot == -1) return;
  if (slot < 0 || slot >= n_slots) {
    if (lane == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  // Rows beyond the request's hold (f, i) = (0, -inf), which leaves m as it is.
  constexpr int kRows = 8;
  float m = m_state[(size_t)slot * H + h];
  float gi[kRows], gf[kRows], gi_next[kRows], gf_next[kRows];
  auto load = [&](int first, float (&to_i)[kRows], float (&to_f)[kRows]) {
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int row = first + lane * kRows + k;
      const bool in = row < n;
      to_i[k] = in ? gates[(size_t)(t0 + row) * 2 * H + h] : -INFINITY;
      to_f[k] = in ? gates[(size_t)(t0 + row) * 2 * H + H + h] : 0.f;
    }
  };
  load(0, gi, gf);
  for (int c = 0; c < n; c += 32 * kRows) {
    load(c + 32 * kRows, gi_next, gf_next);
    const float m_step = m;
    float mine = m, first = 0.f;      // m before the lane's rows; after its first row
    if (in_order) {
      for (int l = 0; l < 32 && c + l * kRows < n; ++l) {
        if (lane >= l) mine = m;
        float walked = m;
#pragma unroll
        for (int k = 0; k < kRows; ++k) walked = fmaxf(gf[k] + walked, gi[k]);
        m = __shfl_sync(0xffffffffu, walked, l);
      }
    } else {
      float f_all = 0.f, i_all = -INFINITY;      // the lane's rows together, then the rows of all lanes up to it
#pragma unroll
      for (int k = 0; k < kRows; ++k) f_all += gf[k], i_all = fmaxf(i_all + gf[k], gi[k]);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float f_left = __shfl_up_sync(0xffffffffu, f_all, o), i_left = __shfl_up_sync(0xffffffffu, i_all, o);
        if (lane >= o) i_all = fmaxf(i_left + f_all, i_all), f_all += f_left;
      }
      const float f_before = __shfl_up_sync(0xffffffffu, f_all, 1), i_before = __shfl_up_sync(0xffffffffu, i_all, 1);
      if (lane > 0) mine = fmaxf(f_before + m, i_before);
    }
#pragma unroll
    for (int k = 0; k < kRows; ++k) {
      const int row = c + lane * kRows + k;
      const float carried = gf[k] + mine;
      mine = fmaxf(carried, gi[k]);
      if (k == 0) first = mine;
      if (row < n) {
        float* g = gates + (size_t)(t0 + row) * 2 * H;
        if (k > 0) g[h] = expf(carried - mine);      // decay of the state
        g[H + h] = expf(gi[k] - mine);               // scale of the new key
        m_out[(size_t)(t0 + row) * H + h] = mine;
      }
    }
    const float left = __shfl_up_sync(0xffffffffu, mine, 1);
    if (c + lane * kRows < n)
      gates[(size_t)(t0 + c + lane * kRows) * 2 * H + h] = expf(gf[0] + (lane == 0 ? m_step : left) - first);
    if (!in_order) m = __shfl_sync(0xffffffffu, mine, min(31, (n - 1 - c) / kRows));      // after the last of these rows
#pragma unroll
    for (int k = 0; k < kRows; ++k) gi[k] = gi_next[k], gf[k] = gf_next[k];
  }
  if (write && lane == 0) m_state[(size_t)slot * H + h] = m;
  pdl_trigger();
}

// One warp per (row, head).
template <typename T>
__global__ void __launch_bounds__(kThreads) memory_finish_kernel(T* __restrict__ out, int ld_out,
                                                                 const float* __restrict__ o, const float* __restrict__ m,
                                                                 const float* __restrict__ gate, int ld_g,
                                                                 const T* __restrict__ w, int tokens, int H, int V,
                                                                 int vpad, float q_scale, float floor_, float eps,
                                                                 float mult, const int* __restrict__ row_req,
                                                                 const int* __restrict__ state_slot) {
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long pair = (long long)blockIdx.x * (kThreads / 32) + warp;
  if (pair >= (long long)tokens * H) return;
  const int t = (int)(pair / H), h = (int)(pair - (long long)t * H);
  if (state_slot[row_req[t]] == -1) {      // a row of padding: the recurrence left nothing for it
    for (int e = lane; e < V; e += 32) out[(size_t)t * ld_out + h * V + e] = from_f32<T>(0.f);
    return;
  }
  const float* oh = o + ((size_t)t * H + h) * vpad;
  const float nq = oh[V] * q_scale;
  const float den = fmaxf(fabsf(nq), expf(-m[(size_t)t * H + h])) + floor_;
  float ss = 0.f;
  for (int e = lane; e < V; e += 32) {
    const float y = oh[e] * q_scale / den;
    ss += y * y;
  }
  ss = warp_sum(ss);
  const float inv = 1.0f / sqrtf(ss / (float)V + eps);
  for (int e = lane; e < V; e += 32) {
    const int c = h * V + e;
    const float y = oh[e] * q_scale / den * inv * to_f32(w[c]);
    const float gz = gate[(size_t)t * ld_g + c];
    out[(size_t)t * ld_out + c] = from_f32<T>(y / (1.f + expf(-gz)) * mult);
  }
}
}  // namespace

// gates [tokens, 2, H] (log input gate, log forget gate), v_out [tokens, H * vpad].
LAB_EXPORT int lab_memory_gates(float* gates, float* v_out, const float* proj, int ld, int v_at, int i_at, int f_at,
                                const void* b_i, const void* b_f, int tokens, int H, int V, int vpad, float cap, int dtype,
                                cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (H <= 0 || V <= 0 || vpad <= V || !(cap > 0.f)) return (int)cudaErrorInvalidValue;
  GateParams p;
  p.proj = proj; p.ld = ld; p.v_at = v_at; p.i_at = i_at; p.f_at = f_at; p.H = H; p.V = V; p.vpad = vpad; p.cap = cap;
  if (dtype == LAB_F32)
    lab_launch(memory_gates_kernel<float>, dim3(tokens), dim3(kThreads), 0, stream, gates, v_out, (const float*)b_i,
               (const float*)b_f, p);
  else
    lab_launch(memory_gates_kernel<__nv_bfloat16>, dim3(tokens), dim3(kThreads), 0, stream, gates, v_out,
               (const __nv_bfloat16*)b_i, (const __nv_bfloat16*)b_f, p);
  LAB_LAUNCH_CHECK();
}

// gates [tokens, 2, H]: in, the log gates; out, the decay and the key's scale of every row.  m_out [tokens, H].
LAB_EXPORT int lab_memory_stabilize(float* gates, float* m_out, float* m_state, const int* q_start, const int* state_slot,
                                    int requests, int n_slots, int H, int write, int in_order, cudaStream_t stream) {
  if (requests <= 0) return 0;
  // A warp's loads and stores touch a sector a lane each, so eight warps of a CTA wait for one another's; a CTA a warp while
  // there are few of them (28 of 1,000 rows 32 us in CTAs of eight, 7 so).
  const int warps = requests * H <= 4 * lab_sm_count() ? 1 : kThreads / 32;
  lab_launch(memory_stabilize_kernel, dim3((requests * H + warps - 1) / warps), dim3(32 * warps), 0, stream, gates, m_out,
             m_state, q_start, state_slot, requests, n_slots, H, write, in_order);
  LAB_LAUNCH_CHECK();
}

LAB_EXPORT int lab_memory_finish(void* out, int ld_out, const float* o, const float* m, const float* gate, int ld_g,
                                 const void* w, int tokens, int H, int V, int vpad, float q_scale, float floor_, float eps,
                                 float mult, const int* row_req, const int* state_slot, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  const long long pairs = (long long)tokens * H;
  const int blocks = (int)((pairs + kThreads / 32 - 1) / (kThreads / 32));
  if (dtype == LAB_F32)
    lab_launch(memory_finish_kernel<float>, dim3(blocks), dim3(kThreads), 0, stream, (float*)out, ld_out, o, m, gate, ld_g,
               (const float*)w, tokens, H, V, vpad, q_scale, floor_, eps, mult, row_req, state_slot);
  else
    lab_launch(memory_finish_kernel<__nv_bfloat16>, dim3(blocks), dim3(kThreads), 0, stream, (__nv_bfloat16*)out, ld_out,
               o, m, gate, ld_g, (const __nv_bfloat16*)w, tokens, H, V, vpad, q_scale, floor_, eps, mult, row_req, state_slot);
  LAB_LAUNCH_CHECK();
}
