// Plain attention over the paged cache: one kernel for any number of new tokens per
// request (whole prompts, portions, single decoded tokens), any head size that is a
// multiple of 8 up to 256, any number of heads and groups, with or without a window.
// It is the attention of the 32-bit path and the yardstick of the tensor-core kernels.
//
// Keys are cut into chunks of 32 by absolute position, one key per lane; a few warps take the chunks in turn, each
// with a running (max, sum, accumulator) in 32-bit, merged at the end in a fixed order.
// The partition depends only on the query's position, so the result for a position is
// the same whatever else is in the batch and however the prompt was cut.  Two kernels: tiles of query rows whose keys
// and values wait in shared memory (heads whose rows are whole 16-byte units), and one block per (query row, head).
//
// Formulas: rust/engine/src/runner/model/qwen2/kernels.rs:702-853 (scores scaled by
// 1/sqrt(d), mask key <= query, online softmax with max/sum/accumulator in 32-bit,
// o = acc / sum), 898-942 (merge of partial softmax states).  The window (keys with
// query - key < window; a negative `window` means chunks of that many positions, see
// `lab_first_key`) is this engine's addition, and so are two options of a window: `keep_first` (the first
// that many positions stay visible to every later query, at their true positions) and `sink` (1: one is
// added to the softmax's denominator, a key with score 0 and no value; with `sinks`, a number per query head,
// exp(sinks[h]) instead), and `dist_bias` [n_q, bias_len]: a number per head and distance query - key that is
// added to the scaled score, distances from bias_len - 1 on sharing the last entry.  `softcap` c > 0: the scaled score
// s becomes c * tanh(s / c) first.  `out_f32`: the output is 32-bit whatever T is.
#include <type_traits>

#include "common.cuh"

namespace {
constexpr int WARPS = 4;
constexpr int MAX_DPL = 8;  // dims per lane: head sizes up to 256

template <typename T>
__global__ void __launch_bounds__(WARPS * 32) attention_plain_kernel(
    void* __restrict__ out, int out_stride, const T* __restrict__ q, int q_stride, const T* __restrict__ cache_k,
    const T* __restrict__ cache_v, const int* __restrict__ row_req, const int* __restrict__ row_pos,
    const int* __restrict__ block_table, int max_blocks, int n_q, int n_kv, int d, int page_size, int num_pages,
    int window, float scale, int keep_first, int sink, const float* __restrict__ sinks,
    const float* __restrict__ dist_bias, int bias_len, float softcap, int out_f32) {
  extern __shared__ float smem[];
  pdl_trigger();
  pdl_wait();
  float* qs = smem;                      // [d]
  float* part = smem + d;                // [WARPS][d + 2]
  const int t = blockIdx.x, h = blockIdx.y, kvh = h / (n_q / n_kv);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int req = row_req[t], p = row_pos[t];
  const int* bt = block_table + (size_t)req * max_blocks;

  for (int i = threadIdx.x; i < d; i += blockDim.x) qs[i] = to_f32<T>(q[(size_t)t * q_stride + (size_t)h * d + i]);
  __syncthreads();

  const int first = lab_first_key(p, window);
  float m = -INFINITY, l = 0.f, acc[MAX_DPL];
#pragma unroll
  for (int i = 0; i < MAX_DPL; ++i) acc[i] = 0.f;

  // two runs of keys: the kept first positions that lie before the window (none without one), then the
  // window itself; each run cut into chunks by absolute position
  const int kept_end = window > 0 && keep_first > 0 ? min(keep_first, first) : 0;
  for (int run = kept_end > 0 ? 0 : 1; run < 2; ++run) {
  const int lo = run == 0 ? 0 : first, hi = run == 0 ? kept_end - 1 : p;
  for (int c = lo / 32 + warp; c * 32 <= hi; c += WARPS) {
    const int j = c * 32 + lane;
    const bool valid = j >= lo && j <= hi;
    long long base = -1;
    float s = -INFINITY;
    if (valid) {
      const int page = bt[j / page_size];
      if (page < 0 || page >= num_pages) {
        lab_set_error(LAB_ERR_PAGE_RANGE);
      } else {
        base = (((long long)page * n_kv + kvh) * page_size + (j % page_size)) * d;
        const T* kr = cache_k + base;
        float dot = 0.f;
        for (int i = 0; i < d; ++i) dot = fmaf(qs[i], to_f32<T>(kr[i]), dot);
        s = dot * scale;
        if (softcap > 0.f) s = softcap * tanhf(s / softcap);
        if (dist_bias != nullptr) s += dist_bias[(size_t)h * bias_len + min(p - j, bias_len - 1)];
      }
    }
    const float m_new = fmaxf(m, warp_max(s));
    if (m_new == -INFINITY) continue;  // no readable key in this chunk (same for the whole warp)
    const float pj = (s == -INFINITY) ? 0.f : expf(s - m_new);
    const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
    l = l * corr + warp_sum(pj);
#pragma unroll
    for (int i = 0; i < MAX_DPL; ++i) acc[i] *= corr;
    for (int jj = 0; jj < 32; ++jj) {
      const float pw = __shfl_sync(0xffffffffu, pj, jj);
      const long long bw = __shfl_sync(0xffffffffu, base, jj);
      if (pw == 0.f || bw < 0) continue;
      const T* vr = cache_v + bw;
#pragma unroll
      for (int i = 0; i < MAX_DPL; ++i) {
        const int dim = lane + 32 * i;
        if (dim < d) acc[i] = fmaf(pw, to_f32<T>(vr[dim]), acc[i]);
      }
    }
    m = m_new;
  }
  }

  float* mine = part + warp * (d + 2);
#pragma unroll
  for (int i = 0; i < MAX_DPL; ++i) {
    const int dim = lane + 32 * i;
    if (dim < d) mine[dim] = acc[i];
  }
  if (lane == 0) {
    mine[d] = m;
    mine[d + 1] = l;
  }
  __syncthreads();
  float big = -INFINITY;
  for (int w = 0; w < WARPS; ++w) big = fmaxf(big, part[w * (d + 2) + d]);
  const float sink_at = sinks != nullptr ? sinks[h] : 0.f;      // the score of the key without a value
  if (sink) big = fmaxf(big, sink_at);
  for (int i = threadIdx.x; i < d; i += blockDim.x) {
    float num = 0.f, den = sink ? expf(sink_at - big) : 0.f;
    for (int w = 0; w < WARPS; ++w) {
      const float mw = part[w * (d + 2) + d];
      const float wt = (mw == -INFINITY) ? 0.f : expf(mw - big);
      num += wt * part[w * (d + 2) + i];
      den += wt * part[w * (d + 2) + d + 1];
    }
    const size_t at = (size_t)t * out_stride + (size_t)h * d + i;
    const float o = den > 0.f ? num / den : 0.f;
    if (out_f32) reinterpret_cast<float*>(out)[at] = o;
    else reinterpret_cast<T*>(out)[at] = from_f32<T>(o);
  }
}

// ---- tiles of query rows ------------------------------------------------------------------------
// A CTA takes 4 RQ WPG rows: neighbouring tokens with the query heads that share one kv head (or some of them, where they
// are more than the tile).  PARTS groups of WPG warps: chunk c of 32 keys goes to group c mod PARTS, whose keys and
// values come to its own buffers by cp.async, the next chunk's keys while the values of this one are used and the other
// way round.  A warp takes 4 RQ rows.  For the scores a lane has four of the rows and every KG-th key of the chunk (two
// products an instruction: sums of even and odd entries apart); the weights are left in shared memory; for the weighted sum it
// has four rows and every KG-th quad of the head's entries.  A row's own arithmetic is the same in every tile and batch.  With the
// requests' first rows (`q_start`) no tile holds rows of two requests: a CTA finds its request by a scan over their
// numbers of tiles, and single tokens beside a prompt's portion are walked side by side.  Without, rows of another request
// in the tile take a pass of their own, after the first.
//
// What bounds it: the multiply-adds (a quarter of the time of 2,000 rows) and what goes around them, the loads of their operands
// from shared memory, exponentials and hand-overs; a lane with one row and key (or entry pair) of eight loaded twice as much and
// looked at every value for infinities.  The other kernel's block per (row, head) reads a row's keys and values once per head
// and row.  Measured on a B200, 32-bit, 14 query and 2 kv heads of 64 (us; the former lanes, then the other kernel in brackets):
// a prompt of 517 43 (54, 560), two of 1,000 208 (299), 8 single tokens after 520 27 (36, 57), where a row's chain of chunks
// bounds it; 12 and 2 heads of 128, 300 rows after 500 131 (177, 1,330).

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool has) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(has ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ float2 load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load2(const __nv_bfloat16* p) {
  const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
}

struct RowsParams {
  void* out;
  const void* q;
  const void* cache_k;
  const void* cache_v;
  const int* row_req;
  const int* row_pos;
  const int* block_table;
  const int* q_start;      // [requests + 1], or null
  const float* sinks;
  const float* dist_bias;
  int requests, out_stride, q_stride, max_blocks, tokens, n_q, n_kv, d, page_size, num_pages, window, keep_first, sink, bias_len,
      out_f32, tile_tokens, head_tiles;      // tokens of a tile; tiles that share a token's heads
  float scale, softcap;
};

template <typename T> __host__ __device__ constexpr int rows_ld(int d) { return d + 16 / (int)sizeof(T); }
template <typename T> static int rows_smem(int d, int parts, int wpg, int rw) {
  return 4 * rw * wpg * d + (int)sizeof(T) * parts * 2 * 32 * rows_ld<T>(d) + 4 * parts * wpg * 32 * (rw + 4);
}

template <typename T, int D, int PARTS, int WPG, int RQ>
__global__ void __launch_bounds__(PARTS * 32 * WPG, D == 64 || (D == 128 && RQ == 2) ? 16 / (PARTS * WPG) : 1) attention_rows_kernel(RowsParams p) {
  extern __shared__ __align__(16) char ap_smem[];
  constexpr int RW = 4 * RQ, R = RW * WPG, NT = PARTS * 32 * WPG;
  constexpr int KG = 32 / RQ, KPL = 32 / KG;                        // key groups, a lane's keys of a chunk
  constexpr int DP = ((D ? D : 256) + 4 * KG - 1) / (4 * KG);       // a lane's quads of a head's entries
  constexpr int WLD = RW + 4;                                       // floats between two keys' weights
  const int d = D ? D : p.d, ld = rows_ld<T>(d);
  float* qs = reinterpret_cast<float*>(ap_smem);                                       // [R][d]
  T* kv = reinterpret_cast<T*>(ap_smem + 4 * R * d);                                   // [PARTS][keys, values][32][ld]
  float* weights = reinterpret_cast<float*>(kv + PARTS * 2 * 32 * ld);                 // [PARTS][WPG][32][WLD]
  __shared__ int s_req[R], s_pos[R];
  pdl_trigger();
  const int tid = threadIdx.x, lane = tid & 31, part = tid / (32 * WPG), warp = (tid >> 5) % WPG;
  const int kvh = blockIdx.y, group = p.n_q / p.n_kv;
  const int tile = gridDim.x - 1 - blockIdx.x;      // the last rows see the most keys: they go first
  int t0 = tile / p.head_tiles * p.tile_tokens, t_end = p.tokens;
  const int h0 = tile % p.head_tiles * R, heads = min(R, group - h0);      // of a token in this tile
  pdl_wait();
  if (p.q_start != nullptr) {
    int left = tile / p.head_tiles;      // tiles of tokens before this one, of requests that have not been passed
    t0 = t_end;
    for (int q0 = 0; q0 < p.requests; q0 += 32) {      // (the same in every warp)
      const int q = q0 + lane, first = q < p.requests ? p.q_start[q] : 0, rows = q < p.requests ? p.q_start[q + 1] - first : 0;
      const int tiles = (rows + p.tile_tokens - 1) / p.tile_tokens;
      int upto = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      const unsigned there = __ballot_sync(0xffffffffu, upto > left);
      if (there != 0u) {
        const int at = __ffs(there) - 1;
        t0 = __shfl_sync(0xffffffffu, first + (left - (upto - tiles)) * p.tile_tokens, at);
        t_end = min(t_end, __shfl_sync(0xffffffffu, first + rows, at));
        break;
      }
      left -= __shfl_sync(0xffffffffu, upto, 31);
    }
    if (t0 >= t_end) return;      // a tile more than there are
  }
  auto token_of = [&](int r) { return t0 + r / heads; };
  auto head_of = [&](int r) { return kvh * group + h0 + r % heads; };
  for (int r = tid; r < R; r += NT) {
    const int t = token_of(r);
    const bool has = r < heads * p.tile_tokens && t < t_end;
    s_req[r] = has ? p.row_req[t] : -1;
    s_pos[r] = has ? p.row_pos[t] : -1;
  }
  __syncthreads();
  for (int i = tid; i < R * d; i += NT) {
    const int r = i / d;
    qs[i] = s_req[r] >= 0 ? to_f32<T>(static_cast<const T*>(p.q)[(size_t)token_of(r) * p.q_stride + (size_t)head_of(r) * d + i % d]) : 0.f;
  }
  __syncthreads();

  T* keys = kv + (size_t)part * 2 * 32 * ld;
  T* values = keys + 32 * ld;
  float* mine = weights + (part * WPG + warp) * 32 * WLD;
  const int rq = lane / KG, kg = lane % KG;      // this lane's rows 4 rq .. of the warp's, its group
  const float* qw = qs + (warp * RW + 4 * rq) * d;
  auto group_sync = [&]() {      // the warps of this group
    if (WPG == 1) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + part), "r"(32 * WPG) : "memory");
  };

  for (int r0 = 0; r0 < R && s_req[r0] >= 0;) {
    // the rows of one request: [r0, r1)
    const int req = s_req[r0];
    int r1 = r0, p_max = -1, lo_min = 0x7fffffff, kept_max = 0;
    for (; r1 < R && s_req[r1] == req; ++r1) {
      const int first = lab_first_key(s_pos[r1], p.window);
      p_max = max(p_max, s_pos[r1]);
      lo_min = min(lo_min, first);
      if (p.window > 0 && p.keep_first > 0) kept_max = max(kept_max, min(p.keep_first, first));
    }
    const int* bt = p.block_table + (size_t)req * p.max_blocks;
    const int last = p_max < 0 ? -1 : p_max / 32;      // (a row of padding sees nothing)
    // chunks that no row sees lie between the kept first positions and the window
    auto settle = [&](int c) {
      if (c * 32 >= kept_max && c < lo_min / 32) c += (lo_min / 32 - c + PARTS - 1) / PARTS * PARTS;
      return c;
    };
    // where key 32 c + lane lies, or -1
    auto place = [&](int c) -> long long {
      const int j = c * 32 + lane;
      if (c > last || j > p_max) return -1;
      const bool seen = j >= lo_min || j < kept_max;
      if (!seen) return -1;
      const int page = bt[j / p.page_size];
      if (page < 0 || page >= p.num_pages) {
        lab_set_error(LAB_ERR_PAGE_RANGE);
        return -1;
      }
      return (((long long)page * p.n_kv + kvh) * p.page_size + j % p.page_size) * d;
    };
    const int units = d * (int)sizeof(T) / 16;
    auto fetch = [&](T* to, const void* cache, long long base, bool any) {
      if (any) {
        // a warp brings 32 / WPG rows, its lanes units side by side
        for (int e = lane; e - lane < 32 / WPG * units; e += 32) {
          const int row = e / units, u = e - row * units;
          const bool in = row < 32 / WPG;
          const long long at = __shfl_sync(0xffffffffu, base, (warp * (32 / WPG) + row) & 31);
          if (in)
            cp_async16(to + (warp * (32 / WPG) + row) * ld + u * (16 / (int)sizeof(T)),
                       static_cast<const T*>(cache) + (at < 0 ? 0 : at) + u * (16 / (int)sizeof(T)), at >= 0);
        }
      }
      cp_async_commit();
    };

    float m[4], l[4][KPL];
    unsigned long long acc[4][DP][2];
    // An infinity or NaN among the values counts for the rows that give it a weight only.  The first pass does not look; if a
    // sum is not finite in the end, a second one leaves terms of weight zero out (finite ones add nothing either way).
    for (bool guarded = false;; guarded = true) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
#pragma unroll
        for (int k = 0; k < KPL; ++k) l[i][k] = 0.f;
#pragma unroll
        for (int u = 0; u < DP; ++u) acc[i][u][0] = acc[i][u][1] = 0ull;
      }
      int c = settle(part);
      long long base = place(c);
      fetch(keys, p.cache_k, base, c <= last);
      fetch(values, p.cache_v, base, c <= last);
      while (c <= last) {
        const int cn = settle(c + PARTS);
        const long long base_n = place(cn);
        cp_async_wait<1>();
        group_sync();
        const unsigned there = __ballot_sync(0xffffffffu, base >= 0);      // the chunk's keys that may be read
        // scores of the lane's rows with its keys; sums of even and odd entries apart
        unsigned long long dot[4][KPL];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int k = 0; k < KPL; ++k) dot[i][k] = 0ull;
        const T* kr = keys + kg * ld;
#pragma unroll 2
        for (int e = 0; e < d; e += 4) {
          unsigned long long k_lo[KPL], k_hi[KPL];
#pragma unroll
          for (int k = 0; k < KPL; ++k) {
            const float4 kq = load4(kr + k * KG * ld + e);
            k_lo[k] = pair_of(kq.x, kq.y), k_hi[k] = pair_of(kq.z, kq.w);
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qw + i * d + e);
#pragma unroll
            for (int k = 0; k < KPL; ++k) fma_pair(dot[i][k], qv.x, k_lo[k]);
#pragma unroll
            for (int k = 0; k < KPL; ++k) fma_pair(dot[i][k], qv.y, k_hi[k]);
          }
        }
        group_sync();
        fetch(keys, p.cache_k, base_n, cn <= last);      // the keys' buffer is free
        float w[KPL][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = warp * RW + 4 * rq + i, pos = s_pos[r];
          const int first = lab_first_key(pos, p.window);
          const int kept = p.window > 0 && p.keep_first > 0 ? min(p.keep_first, first) : 0;
          float s[KPL], top = -INFINITY;
#pragma unroll
          for (int k = 0; k < KPL; ++k) {
            const int key = kg + KG * k, j = c * 32 + key;
            s[k] = -INFINITY;
            if (r >= r0 && r < r1 && (there >> key & 1u) != 0u && j <= pos && (j >= first || j < kept)) {
              s[k] = (low_of(dot[i][k]) + high_of(dot[i][k])) * p.scale;
              if (p.softcap > 0.f) s[k] = p.softcap * tanhf(s[k] / p.softcap);
              if (p.dist_bias != nullptr) s[k] += p.dist_bias[(size_t)head_of(r) * p.bias_len + min(pos - j, p.bias_len - 1)];
            }
            top = fmaxf(top, s[k]);
          }
#pragma unroll
          for (int o = KG / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
          const float m_new = fmaxf(m[i], top);
#pragma unroll
          for (int k = 0; k < KPL; ++k) w[k][i] = 0.f;
          if (m_new != -INFINITY) {      // (else no readable key so far)
            const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
#pragma unroll
            for (int k = 0; k < KPL; ++k) {
              w[k][i] = s[k] == -INFINITY ? 0.f : expf(s[k] - m_new);
              l[i][k] = l[i][k] * corr + w[k][i];
            }
            const unsigned long long cc = pair_of(corr, corr);
#pragma unroll
            for (int u = 0; u < DP; ++u) {
              asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[i][u][0]) : "l"(cc));
              asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[i][u][1]) : "l"(cc));
            }
            m[i] = m_new;
          }
        }
#pragma unroll
        for (int k = 0; k < KPL; ++k) store4(mine + (kg + KG * k) * WLD + 4 * rq, make_float4(w[k][0], w[k][1], w[k][2], w[k][3]));
        cp_async_wait<1>();
        group_sync();
        // the weighted sum: a key's weights of the lane's rows, its quads kg, kg + KG, .. of the entries
        auto weighted = [&](auto guard) {
#pragma unroll 4
          for (int jj = 0; jj < 32; ++jj) {
            const float4 w4 = load4(mine + jj * WLD + 4 * rq);
            const float wt[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int u = 0; u < DP; ++u) {
              const int e = 4 * (kg + KG * u);
              if (D % (4 * KG) != 0 || D == 0) {
                if (e >= d) break;
              }
              const float4 v = load4(values + jj * ld + e);
              const unsigned long long v_lo = pair_of(v.x, v.y), v_hi = pair_of(v.z, v.w);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                if (decltype(guard)::value && wt[i] == 0.f) continue;
                const unsigned long long ww = pair_of(wt[i], wt[i]);
                fma_pair(acc[i][u][0], ww, v_lo);
                fma_pair(acc[i][u][1], ww, v_hi);
              }
            }
          }
        };
        if (guarded) weighted(std::true_type{});
        else weighted(std::false_type{});
        group_sync();
        fetch(values, p.cache_v, base_n, cn <= last);
        c = cn;
        base = base_n;
      }
      bool finite = true;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int u = 0; u < DP; ++u)
          finite &= isfinite(low_of(acc[i][u][0])) && isfinite(high_of(acc[i][u][0])) && isfinite(low_of(acc[i][u][1])) &&
                    isfinite(high_of(acc[i][u][1]));
      cp_async_wait<0>();
      if (!__syncthreads_or(!finite && !guarded)) break;      // every buffer has been read
    }
    float* results = reinterpret_cast<float*>(kv);      // the parts' results take the buffers' place: [PARTS][R][d + 2]
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float* to = results + (part * R + warp * RW + 4 * rq + i) * (d + 2);
      // (the order of a sum over 32 lanes with a key each: half with half)
#pragma unroll
      for (int o = KPL / 2; o > 0; o /= 2)
#pragma unroll
        for (int k = 0; k < o; ++k) l[i][k] += l[i][k + o];
      float all = l[i][0];
#pragma unroll
      for (int o = KG / 2; o > 0; o >>= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
      if (kg == 0) to[d] = m[i], to[d + 1] = all;
#pragma unroll
      for (int u = 0; u < DP; ++u) {
        const int e = 4 * (kg + KG * u);
        if (e >= d) break;
        to[e] = low_of(acc[i][u][0]), to[e + 1] = high_of(acc[i][u][0]);
        to[e + 2] = low_of(acc[i][u][1]), to[e + 3] = high_of(acc[i][u][1]);
      }
    }
    __syncthreads();
    for (int x = tid; x < (r1 - r0) * d; x += NT) {
      const int r = r0 + x / d, i = x % d, h = head_of(r);
      const float sink_at = p.sinks != nullptr ? p.sinks[h] : 0.f;      // the score of the key without a value
      float big = -INFINITY;
#pragma unroll
      for (int w = 0; w < PARTS; ++w) big = fmaxf(big, results[(w * R + r) * (d + 2) + d]);
      if (p.sink) big = fmaxf(big, sink_at);
      float num = 0.f, den = p.sink ? expf(sink_at - big) : 0.f;
#pragma unroll
      for (int w = 0; w < PARTS; ++w) {
        const float* from = results + (w * R + r) * (d + 2);
        const float wt = from[d] == -INFINITY ? 0.f : expf(from[d] - big);
        num += wt * from[i];
        den += wt * from[d + 1];
      }
      const size_t at = (size_t)token_of(r) * p.out_stride + (size_t)h * d + i;
      const float o = den > 0.f ? num / den : 0.f;
      if (p.out_f32) static_cast<float*>(p.out)[at] = o;
      else static_cast<T*>(p.out)[at] = from_f32<T>(o);
    }
    __syncthreads();
    r0 = r1;
  }
}

template <typename T, int D, int PARTS, int WPG, int RQ>
int launch_rows(RowsParams p, cudaStream_t stream) {
  const int smem = rows_smem<T>(p.d, PARTS, WPG, 4 * RQ);
  static LabShared granted;
  const cudaError_t e = lab_allow_shared(granted, (const void*)attention_rows_kernel<T, D, PARTS, WPG, RQ>, smem);
  if (e != cudaSuccess) return (int)e;
  if (p.tile_tokens == 1) p.q_start = nullptr;
  // with the requests' borders: every request may end in a tile that is not full
  const long long more = p.q_start != nullptr ? (long long)p.requests * (p.tile_tokens - 1) : p.tile_tokens - 1;
  const long long tiles = (p.tokens + more) / p.tile_tokens * p.head_tiles;
  return (int)lab_launch(attention_rows_kernel<T, D, PARTS, WPG, RQ>, dim3((unsigned)tiles, p.n_kv), dim3(PARTS * 32 * WPG),
                         smem, stream, p);
}

// Sixteen rows a CTA halve what it reads, eight give twice the CTAs: sixteen once they fill every multiprocessor twice.  With
// heads of 64 thirty-two, sixteen to a warp, once they fill every multiprocessor four times: fewer leave the long rows' CTAs
// alone at the end.  Measured (us, 32 / 16 rows, 14 and 2 heads): one prompt of 1,200 143 / 162, 1,600 246 / 268, 800 85 / 84,
// 517 59 / 43, two of 1,000 208 / 234, three of 400 85 / 81, eight of 250 120 / 127.  (Heads of 128 have no tile of thirty-two: a
// lane's sums of four rows by sixteen entries and four keys' products would take all the registers that four CTAs leave.)
template <typename T>
int pick_rows(RowsParams p, bool single, cudaStream_t stream) {
  const int group = p.n_q / p.n_kv;
  auto shape = [&](int rows) {
    p.tile_tokens = single || group >= rows ? 1 : rows / group;
    p.head_tiles = (group + rows - 1) / rows;
    return ((long long)p.tokens + p.tile_tokens - 1) / p.tile_tokens * p.head_tiles * p.n_kv;
  };
  if (p.d == 64 && shape(32) >= 4 * lab_sm_count()) return launch_rows<T, 64, 4, 2, 4>(p, stream);
  const bool wide = shape(16) >= 2 * lab_sm_count();
  if (!wide) shape(8);
  if (p.d == 64) return wide ? launch_rows<T, 64, 4, 2, 2>(p, stream) : launch_rows<T, 64, 4, 1, 2>(p, stream);
  if (p.d == 128) return wide ? launch_rows<T, 128, 4, 2, 2>(p, stream) : launch_rows<T, 128, 4, 1, 2>(p, stream);
  if (p.d < 128) return wide ? launch_rows<T, 0, 4, 2, 2>(p, stream) : launch_rows<T, 0, 4, 1, 2>(p, stream);
  return wide ? launch_rows<T, 0, 2, 2, 2>(p, stream) : launch_rows<T, 0, 2, 1, 2>(p, stream);
}
}  // namespace

// `single`: no request brings more than one row (rows of one token then make up a tile).  q_start: the requests' first
// rows, and the number of all rows behind them, or null; then no tile takes rows of two requests.
LAB_EXPORT int lab_attention_plain(void* out, int out_stride, const void* q, int q_stride, const void* cache_k,
                                   const void* cache_v, const int* row_req, const int* row_pos, const int* block_table,
                                   int max_blocks, int tokens, int n_q, int n_kv, int d, int page_size, int num_pages,
                                   int window, float scale, int keep_first, int sink, const float* sinks,
                                   const float* dist_bias, int bias_len, float softcap, int out_f32, int single,
                                   const int* q_start, int requests, int dtype, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (d > 32 * MAX_DPL || d <= 0 || n_q % n_kv || (dist_bias != nullptr && bias_len < 1)) return (int)cudaErrorInvalidValue;
  if (sinks != nullptr) sink = 1;
  if (d % (dtype == LAB_F32 ? 4 : 8) == 0 && (((uintptr_t)cache_k | (uintptr_t)cache_v) & 15) == 0 && n_kv <= 65535) {
    const RowsParams p{out, q, cache_k, cache_v, row_req, row_pos, block_table, requests > 1 ? q_start : nullptr, sinks,
                       dist_bias, requests, out_stride, q_stride, max_blocks, tokens, n_q, n_kv, d, page_size, num_pages, window, keep_first, sink, bias_len,
                       out_f32, 1, 1, scale, softcap};
    return dtype == LAB_F32 ? pick_rows<float>(p, single != 0, stream) : pick_rows<__nv_bfloat16>(p, single != 0, stream);
  }
  dim3 grid(tokens, n_q);
  const size_t smem = (size_t)(d + WARPS * (d + 2)) * sizeof(float);
  if (dtype == LAB_F32)
    return (int)lab_launch(attention_plain_kernel<float>, grid, dim3(WARPS * 32), smem, stream, out, out_stride,
                           (const float*)q, q_stride, (const float*)cache_k, (const float*)cache_v, row_req, row_pos,
                           block_table, max_blocks, n_q, n_kv, d, page_size, num_pages, window, scale, keep_first,
                           sink, sinks, dist_bias, bias_len, softcap, out_f32);
  return (int)lab_launch(attention_plain_kernel<__nv_bfloat16>, grid, dim3(WARPS * 32), smem, stream,
                         out, out_stride, (const __nv_bfloat16*)q, q_stride,
                         (const __nv_bfloat16*)cache_k, (const __nv_bfloat16*)cache_v, row_req, row_pos, block_table,
                         max_blocks, n_q, n_kv, d, page_size, num_pages, window, scale, keep_first, sink, sinks, dist_bias,
                         bias_len, softcap, out_f32);
}
