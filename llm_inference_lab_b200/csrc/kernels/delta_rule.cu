// Generalized delta rule: a recurrent mixer whose state per head is a matrix S [key channel,
// value channel] in 32-bit floats, carried from token to token:
//
//   S <- diag(w) S  -  (a * u) (u^T S)  +  k v^T          (both products read the old S)
//   o  = S^T r
//
// with per-channel decay w = exp(-rate * sigmoid(d)), removal rate a = sigmoid(.), and the unit key
// u = k / sqrt(sum k^2 + 1e-6).  The kernel takes the projections r, k, v, the gate's and the two
// rates' pre-activations in 32-bit, forms every quantity of the recurrence in 32-bit, walks a
// request's tokens in order, divides each head's o by its root mean square, multiplies by a weight
// and by sigmoid(gate) and rounds to the storage type for the output projection.
//
// One CTA per (head, request, slice of CS columns of S).  Built per head size D (LAB_HEAD_DIM).  The
// columns of S are independent of one another, and so are its rows within a token, so a column is shared
// out over G threads (4 where D allows): thread g keeps the rows g * SL .. g * SL + SL - 1 of column j in
// registers, reads its share of each vector with consecutive 16-byte loads (a vector lies row block by
// row block with four floats of padding between the blocks, so the G threads of a column hit different
// banks, and lanes of other columns read the same addresses), and the sums over a column are finished by
// log2(G) shuffles.  (Blocks interleaved over the threads, without padding, are as free of conflicts and
// measured slower: 0.90 against 0.75 ms for 2,048 tokens of one request.)  What bounds the walk is the chain of dependent
// instructions one warp has per token (measured with the kernel's own clock: 540 cycles a token with
// 4 threads a column and 16 rows each, an entry an instruction, and every token's loads in front of its arithmetic;
// now two rows an instruction, and a vector's share of the next token is asked for as soon as this token's is used),
// and a head's columns are shared out over D / CS CTAs so that
// no scheduler holds more than one such chain.  (Measured with the mixer around it, 14 heads of 64: one request of 2,048
// tokens 517 us against 632 in the earlier form, 300 tokens 98 against 120, three of 500 201 against 218.)
// Tokens are taken in chunks:
// a chunk's records are brought to shared memory by cp.async into the buffer that is not being walked.
// Three kernels: a first one, parallel over tokens, forms what does not depend on the state (decays,
// rates, unit keys); the walk; a third, parallel over tokens, divides each head's raw output by its root
// mean square and applies weight and gate.  A step of one token per request (decode) is the same three
// kernels with a chunk of one.
#include <type_traits>

#include "tcgen05.cuh"

#ifndef LAB_HEAD_DIM
#define LAB_HEAD_DIM 64
#endif

namespace {

constexpr int D = LAB_HEAD_DIM;
// threads per column: up to 4, so that every thread has whole blocks of four rows.  (Measured at D = 64,
// 2,048 tokens of one request: 4 threads a column 0.74 ms, 16 threads a column 1.17 ms: a level of
// shuffles costs the walk about as much as 25 rows a thread.)
constexpr int G = D % 16 == 0 ? 4 : D % 8 == 0 ? 2 : 1;
constexpr bool VEC = D % (4 * G) == 0;               // false: one thread a column, one value a load
constexpr int SL = D / G;                            // rows of a column per thread
constexpr int CS = (D % 16 == 0 && D > 16) ? 16 : D;  // columns of S per CTA
constexpr int NS = D / CS;                           // CTAs per head
constexpr int NT = ((CS * G + 31) / 32) * 32;
constexpr int CH = 16;                               // tokens per chunk
static_assert(D >= 4 && D <= 256, "head size of the delta rule kernel: 4 to 256");

__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }

// What the walk reads per token and head is one record, prepared by a kernel that is parallel over
// tokens and copied to shared memory as it is:
//   u, r * w, w, a * u, k   five vectors over the rows of S
//   v                       D values
//   alpha, beta             alpha = r . (a * u), beta = r . k
// With them the output needs only the OLD state:
//   o_j = sum_i r_i S'_ij = (r * w) . S_j  -  alpha (u . S_j)  +  beta v_j
// so a token costs two independent sums over a column of S and one update, of which only one multiply-add
// waits for the sums.  Records of one head lie token after token in global memory: a chunk is one
// contiguous block.  (Loads into registers instead, issued before the walk of the chunk before, held the
// walk's own shared-memory loads back behind them in the load pipe.)
constexpr int PV = 5;
// A vector over the rows of S lies row block by row block: thread g's rows g * SL .. g * SL + SL - 1
// together, then four floats of padding, so that a thread's share is consecutive 16-byte loads and the G
// threads of a column hit different banks.
constexpr int SLP = VEC ? SL + 4 : SL;
constexpr int RL = G * SLP;
constexpr int REC = (PV * RL + D + 2 + 3) / 4 * 4;      // floats of a record
constexpr int OFF_V = PV * RL, OFF_AB = PV * RL + D;
__device__ __forceinline__ int at_row(int i) { return (i / SL) * SLP + (i % SL); }
// row of S that thread g holds in register ii
__device__ __forceinline__ int row_of(int g, int ii) { return g * SL + ii; }

struct DeltaParams {
  float* out;           // [tokens, heads * D]: each head's raw output o = S^T r
  const float* rec;     // [heads][tokens][REC]
  int tokens;
  float* state;         // [slots, heads, D, D] floats
  const int* q_start;   // [requests + 1]
  const int* state_slot;
  int heads, n_slots, write;
};

struct DeltaShared {
  float rec[2][CH][REC];
};

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

constexpr int SP = (SL + 1) / 2;      // pairs of rows a thread keeps (an odd last row beside a zero)

// A thread's SL values of one vector of D values in shared memory, in pairs.
__device__ __forceinline__ void load_rows(f32x2 (&dst)[SP], const float* vec, int g) {
  if constexpr (VEC) {
#pragma unroll
    for (int q = 0; q < SL / 4; ++q) {
      const ulonglong2 t = reinterpret_cast<const ulonglong2*>(vec + g * SLP)[q];
      dst[2 * q] = t.x, dst[2 * q + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int ii = 0; ii < SP; ++ii) dst[ii] = pair_of(vec[g * SLP + 2 * ii], 2 * ii + 1 < SL ? vec[g * SLP + 2 * ii + 1] : 0.f);
  }
}

template <typename T>
__global__ void __launch_bounds__(NT) delta_rule_kernel(DeltaParams p) {
  extern __shared__ __align__(16) uint8_t delta_smem[];
  static_assert(REC % 4 == 0 && (!VEC || (SLP % 4 == 0 && RL % 4 == 0)), "16-byte loads");
  DeltaShared& sh = *reinterpret_cast<DeltaShared*>(delta_smem);
  pdl_wait();
  const int h = blockIdx.x, req = blockIdx.y;
  const int tid = threadIdx.x;
  const int j = blockIdx.z * CS + tid / G, g = tid % G;      // this thread's column of S and its rows' block
  const bool live = tid / G < CS;
  const int row0 = p.q_start[req], row1 = p.q_start[req + 1];
  const int slot = p.state_slot[req];
  if (slot == -1) {      // a request of padding (length zero in a padded batch): zeros out, no state
    const int jj = blockIdx.z * CS + tid / G;
    if (tid / G < CS && tid % G == 0)
      for (int t = row0; t < row1; ++t) p.out[(size_t)t * p.heads * D + h * D + jj] = 0.f;
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  float* S_g = p.state + ((size_t)slot * p.heads + h) * D * D;
  f32x2 S[SP];
#pragma unroll
  for (int ii = 0; ii < SP; ++ii)
    S[ii] = pair_of(live ? S_g[(size_t)row_of(g, 2 * ii) * D + j] : 0.f,
                    live && 2 * ii + 1 < SL ? S_g[(size_t)row_of(g, 2 * ii + 1) * D + j] : 0.f);
  const int ld_out = p.heads * D;
  const float* records = p.rec + (size_t)h * p.tokens * REC;

  // chunk c of the request -> buffer c & 1, sixteen bytes a copy
  auto fetch = [&](int t0, int buf) {
    const int n16 = min(CH, row1 - t0) * (REC / 4);
    const float* src = records + (size_t)t0 * REC;
    const uint32_t dst = smem_u32(&sh.rec[buf][0][0]);
    for (int c = tid; c < n16; c += NT) cp_async_16(dst + 16 * c, src + 4 * c);
    cp_async_commit_group();
  };

  fetch(row0, 0);
  int buf = 0;
  for (int t0 = row0; t0 < row1; t0 += CH, buf ^= 1) {
    const int n = min(CH, row1 - t0);
    cp_async_wait_all();
    __syncthreads();       // the chunk has landed for everyone, and the other buffer's readers are done
    if (t0 + CH < row1) fetch(t0 + CH, buf ^ 1);
    // ---- the recurrence, token by token ---------------------------------------------------
    // What does not wait for the sums over the column (w * S + k * v_j) is formed beside them, so that one
    // multiply-add follows the shuffles; the next token's values are asked for where this token's are used up.
    // (With more than 16 rows a thread the registers do not allow it: a token's values are asked for in front.)
    constexpr bool AHEAD = SL <= 16;
    f32x2 u[SP], rw_[SP], w[SP], au[SP], kk[SP];
    float vj, alpha, beta;
    auto load_all = [&](const float* rec) {
      load_rows(u, rec, g);
      load_rows(rw_, rec + RL, g);
      load_rows(w, rec + 2 * RL, g);
      load_rows(kk, rec + 4 * RL, g);
      load_rows(au, rec + 3 * RL, g);
      vj = live ? rec[OFF_V + j] : 0.f, alpha = rec[OFF_AB], beta = rec[OFF_AB + 1];
    };
    if (AHEAD) load_all(sh.rec[buf][0]);
    for (int tok = 0; tok < n; ++tok) {
      if (!AHEAD) load_all(sh.rec[buf][tok]);
      const float* rec = sh.rec[buf][min(tok + 1, n - 1)];
      const float v_now = vj, alpha_now = alpha, beta_now = beta;
      constexpr int NA = AHEAD ? 2 : 1;      // sums side by side (more of them cost more in additions than they hide)
      f32x2 s2[2] = {0ull, 0ull}, r2[2] = {0ull, 0ull};      // zeros
#pragma unroll
      for (int ii = 0; ii < SP; ++ii) {
        s2[ii % NA] = fma2(u[ii], S[ii], s2[ii % NA]);
        r2[ii % NA] = fma2(rw_[ii], S[ii], r2[ii % NA]);
      }
      if (AHEAD) {
        load_rows(u, rec, g);
        load_rows(rw_, rec + RL, g);
        vj = live ? rec[OFF_V + j] : 0.f, alpha = rec[OFF_AB], beta = rec[OFF_AB + 1];
      }
      float sa = low_of(s2[0]) + high_of(s2[0]), rw = low_of(r2[0]) + high_of(r2[0]);
      if (NA == 2) sa += low_of(s2[1]) + high_of(s2[1]), rw += low_of(r2[1]) + high_of(r2[1]);
      const f32x2 vv = pair_of(v_now, v_now);
#pragma unroll
      for (int ii = 0; ii < SP; ++ii) S[ii] = AHEAD ? fma2(kk[ii], vv, mul2(w[ii], S[ii])) : fma2(w[ii], S[ii], mul2(kk[ii], vv));
      if (AHEAD) {
        load_rows(w, rec + 2 * RL, g);
        load_rows(kk, rec + 4 * RL, g);
      }
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        sa += __shfl_xor_sync(0xffffffffu, sa, o);
        rw += __shfl_xor_sync(0xffffffffu, rw, o);
      }
      const f32x2 minus_sa = pair_of(-sa, -sa);
#pragma unroll
      for (int ii = 0; ii < SP; ++ii) S[ii] = fma2(au[ii], minus_sa, S[ii]);
      if (AHEAD) load_rows(au, rec + 3 * RL, g);
      if (live && g == 0) p.out[(size_t)(t0 + tok) * ld_out + h * D + j] = fmaf(beta_now, v_now, fmaf(-alpha_now, sa, rw));
    }
  }
  pdl_trigger();      // (not earlier: the next kernel's blocks would settle beside this one's and slow them down)
  if (p.write && live) {
#pragma unroll
    for (int ii = 0; ii < SL; ++ii) S_g[(size_t)row_of(g, ii) * D + j] = ii % 2 == 0 ? low_of(S[ii / 2]) : high_of(S[ii / 2]);
  }
}

// Per token and head, everything of the recurrence that does not depend on the state, in 32-bit:
// decay w = exp(-rate * sigmoid(d + bias)), removal a = sigmoid(. + bias), unit key u, and the products
// the walk uses.  One CTA per token, a warp per head at a time.
template <typename T>
__global__ void __launch_bounds__(256) delta_prepare_kernel(float* __restrict__ records, int tokens,
                                                            const float* __restrict__ r, const float* __restrict__ k,
                                                            const float* __restrict__ v, const float* __restrict__ a,
                                                            int ld, const float* __restrict__ d, int ld_d,
                                                            const T* __restrict__ d_bias, const T* __restrict__ a_bias,
                                                            int heads, float decay_rate) {
  pdl_wait();
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int h = blockIdx.y * 8 + warp; h < heads; h += 8 * gridDim.y) {
    const size_t at = (size_t)t * ld + h * D;
    float ss = 0.f;
    for (int i = lane; i < D; i += 32) ss += k[at + i] * k[at + i];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss + 1e-6f);
    float* dst = records + ((size_t)h * tokens + t) * REC;
    float al = 0.f, be = 0.f;
    for (int i = lane; i < D; i += 32) {
      const float kk = k[at + i], rr = r[at + i];
      const float w = expf(-decay_rate * sigmoidf_(d[(size_t)t * ld_d + h * D + i] + to_f32(d_bias[h * D + i])));
      const float u = kk * inv, au = sigmoidf_(a[at + i] + to_f32(a_bias[h * D + i])) * u;
      const int ir = at_row(i);
      dst[ir] = u, dst[RL + ir] = rr * w, dst[2 * RL + ir] = w, dst[3 * RL + ir] = au, dst[4 * RL + ir] = kk;
      dst[OFF_V + i] = v[at + i];
      al = fmaf(rr, au, al);
      be = fmaf(rr, kk, be);
    }
    al = warp_sum(al);
    be = warp_sum(be);
    if (lane == 0) dst[OFF_AB] = al, dst[OFF_AB + 1] = be;
  }
  pdl_trigger();      // (not earlier: the walk's few, long blocks would settle unevenly where these leave room first)
}

// ---- portions of a prompt: four tokens in one go ---------------------------------------------------
// Within a block of tokens 0..3 let P_i be the product of the decays up to token i, R_ij that of the decays after token j
// up to token i, and p_i = u_i^T S the old state's part that token i removes.  With the state S before the block
//
//   p_i = (P_{i-1} u_i)^T S + sum_{j<i} (u_i . R_{i-1,j} k_j) v_j - (u_i . R_{i-1,j} a_j u_j) p_j
//   o_i = (P_i r_i)^T S     + sum_{j<=i} (r_i . R_ij k_j) v_j     - (r_i . R_ij a_j u_j) p_j
//   S  <- P_3 S + sum_j (R_3j k_j) v_j^T - (R_3j a_j u_j) p_j^T
//
// which is the recurrence with its sums regrouped: eight independent sums over a column of S, four steps on numbers, one
// update, where there were four dependent rounds.  Products of decays are formed as products, never as quotients, so
// strong decays lose nothing.  A request's blocks start at its first row; rows beyond its last have decay 1 and zeros.
// 32-bit storage keeps the walk token by token: a result must not depend on where a portion starts.
constexpr int BLK = 4;
constexpr int B_DOTS = 8, B_KEYS = 8, B_GONE = 12, B_DECAY = 16, B_VECTORS = 17;      // P u, P r; R k; -R a u; P_3
constexpr int N_PAIR = BLK * (BLK - 1) / 2, N_TRI = BLK * (BLK + 1) / 2;              // j < i and j <= i
// coefficients: u . R k and -u . R a u of the pairs j < i, then a row of r . R k and one of -r . R a u a token (zeros
// beyond j = i)
constexpr int C_UK = 0, C_UA = N_PAIR, C_RK = 2 * N_PAIR, C_RA = C_RK + BLK * BLK, N_COEF = C_RA + BLK * BLK;
static_assert(2 * (N_PAIR + N_TRI) == 32 && N_COEF % 4 == 0, "a lane a sum");
// Eight rows of two columns a thread, so that a whole block's share of the record fits its registers and is asked for a
// block ahead: GB threads a pair of columns.
constexpr bool BLOCKS_BUILT = D == 32 || D == 64 || D == 128 || D == 256;
constexpr int SLB = 8, GB = BLOCKS_BUILT ? D / SLB : 4, SLBP = SLB + 4, RLB = GB * SLBP;      // (padded as above)
constexpr int AT_V = B_VECTORS * RLB, AT_C = AT_V + BLK * D, BREC = AT_C + N_COEF;             // floats of a record
constexpr int BCHUNK = BREC * 4 * 8 <= 64 * 1024 ? 4 : 2;                                      // blocks of a chunk
constexpr int NCOL = 2, BCOLS = 16, BTHREADS = BCOLS / NCOL * GB;
constexpr size_t BSMEM = sizeof(float) * 2 * BCHUNK * BREC + 32;      // two chunks, their barriers, the abort flag

// The place of a request's first block among the records of a head: there are no more than tokens / 4 + requests.
__host__ __device__ __forceinline__ int first_block(int row0, int request) { return row0 / BLK + request; }

// One warp per (block, head): everything of the recurrence that does not depend on the state.  Bound by its writes.
template <typename T>
__global__ void __launch_bounds__(256) delta_prepare_blocks_kernel(float* __restrict__ records, int n_records,
                                                                   const float* __restrict__ r, const float* __restrict__ k,
                                                                   const float* __restrict__ v, const float* __restrict__ a,
                                                                   int ld, const float* __restrict__ d, int ld_d,
                                                                   const T* __restrict__ d_bias, const T* __restrict__ a_bias,
                                                                   const int* __restrict__ q_start, int requests, int heads,
                                                                   float decay_rate) {
  pdl_wait();
  const int lane = threadIdx.x & 31, h = blockIdx.y * 8 + (threadIdx.x >> 5), at = blockIdx.x;
  // the last request whose blocks start at or before this record
  int req = 0;
  for (int r0 = 0; r0 < requests; r0 += 32) {
    const bool before = r0 + lane < requests && first_block(q_start[min(r0 + lane, requests - 1)], r0 + lane) <= at;
    const unsigned all = __ballot_sync(0xffffffffu, before);
    if (all == 0u) break;
    req = r0 + 31 - __clz((int)all);
  }
  const int row0 = q_start[req], t0 = row0 + BLK * (at - first_block(row0, req)), n = min(BLK, q_start[req + 1] - t0);
  if (n > 0 && h < heads) {
    float inv[BLK];
#pragma unroll
    for (int t = 0; t < BLK; ++t) {
      float ss = 0.f;
      for (int i = lane; i < D; i += 32) {
        const float kk = t < n ? k[(size_t)(t0 + t) * ld + h * D + i] : 0.f;
        ss = fmaf(kk, kk, ss);
      }
      inv[t] = 1.0f / sqrtf(warp_sum(ss) + 1e-6f);
    }
    float c[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) c[i] = 0.f;
    float* dst = records + ((size_t)h * n_records + at) * BREC;
    for (int i = lane; i < D; i += 32) {
      const int ch = h * D + i, ir = (i / SLB) * SLBP + i % SLB;
      float w[BLK], u[BLK], au[BLK], kk[BLK], rr[BLK];
#pragma unroll
      for (int t = 0; t < BLK; ++t) {
        w[t] = 1.f, u[t] = au[t] = kk[t] = rr[t] = 0.f;
        float vv = 0.f;
        if (t < n) {
          const size_t from = (size_t)(t0 + t) * ld + ch;
          kk[t] = k[from], rr[t] = r[from], vv = v[from];
          w[t] = expf(-decay_rate * sigmoidf_(d[(size_t)(t0 + t) * ld_d + ch] + to_f32(d_bias[ch])));
          u[t] = kk[t] * inv[t];
          au[t] = -(sigmoidf_(a[from] + to_f32(a_bias[ch])) * u[t]);
        }
        dst[AT_V + t * D + i] = vv;
      }
      float before = 1.f;      // the product of the decays up to the token before
#pragma unroll
      for (int t = 0; t < BLK; ++t) {
        dst[t * RLB + ir] = before * u[t];
        before *= w[t];
        dst[(BLK + t) * RLB + ir] = before * rr[t];
      }
      dst[B_DECAY * RLB + ir] = before;
      // R_{i-1,j} k_j and -R_{i-1,j} a_j u_j for all j < i, then R_3j's; token by token
      float rk[BLK], ra[BLK];
      int pair = 0, tri = 0;
#pragma unroll
      for (int t = 0; t < BLK; ++t) {
#pragma unroll
        for (int j = 0; j < t; ++j, ++pair) {
          c[pair] = fmaf(u[t], rk[j], c[pair]);
          c[N_PAIR + pair] = fmaf(u[t], ra[j], c[N_PAIR + pair]);
        }
        rk[t] = kk[t], ra[t] = au[t];
#pragma unroll
        for (int j = 0; j <= t; ++j, ++tri) {
          if (j < t) rk[j] *= w[t], ra[j] *= w[t];
          c[2 * N_PAIR + tri] = fmaf(rr[t], rk[j], c[2 * N_PAIR + tri]);
          c[2 * N_PAIR + N_TRI + tri] = fmaf(rr[t], ra[j], c[2 * N_PAIR + N_TRI + tri]);
        }
      }
#pragma unroll
      for (int t = 0; t < BLK; ++t) dst[(B_KEYS + t) * RLB + ir] = rk[t], dst[(B_GONE + t) * RLB + ir] = ra[t];
    }
    // 32 sums over the lanes, one of them left in each lane
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float mine = upper ? c[i + o] : c[i], theirs = upper ? c[i] : c[i + o];
        c[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
      }
    }
    float* coef = dst + AT_C;
    if (lane < 2 * N_PAIR) {
      coef[lane] = c[0];
      // (the twelve places beyond the diagonals)
      const int pair = lane % N_PAIR, i = pair < 3 ? 0 : pair < 5 ? 1 : 2, j = pair < 3 ? pair + 1 : pair < 5 ? pair - 1 : 3;
      coef[(lane < N_PAIR ? C_RK : C_RA) + BLK * i + j] = 0.f;
    } else {
      const int tri = (lane - 2 * N_PAIR) % N_TRI, i = tri < 1 ? 0 : tri < 3 ? 1 : tri < 6 ? 2 : 3;
      coef[(lane < 2 * N_PAIR + N_TRI ? C_RK : C_RA) + BLK * i + tri - i * (i + 1) / 2] = c[0];
    }
  }
  pdl_trigger();      // (not earlier: see delta_prepare_kernel)
}

// A thread's eight rows of one vector of a record, in pairs.
__device__ __forceinline__ void load_share(f32x2 (&dst)[SLB / 2], const float* share, int vector) {
#pragma unroll
  for (int q = 0; q < SLB / 4; ++q) {
    const ulonglong2 t = reinterpret_cast<const ulonglong2*>(share + vector * RLB)[q];
    dst[2 * q] = t.x, dst[2 * q + 1] = t.y;
  }
}

__global__ void __launch_bounds__(BTHREADS) delta_blocks_kernel(DeltaParams p, int n_records) {
  extern __shared__ __align__(16) float blocks_smem[];
  pdl_wait();
  const int h = blockIdx.x, req = blockIdx.y, tid = threadIdx.x;
  const int j = blockIdx.z * BCOLS + tid / GB * NCOL, g = tid % GB;      // this thread's first column of S, its share of the rows
  const int row0 = p.q_start[req], rows = p.q_start[req + 1] - row0;
  const int slot = p.state_slot[req];
  if (slot == -1) {      // rows of padding: zeros out, no state
    if (g == 0)
      for (int t = row0; t < row0 + rows; ++t)
        *reinterpret_cast<float2*>(p.out + (size_t)t * p.heads * D + h * D + j) = make_float2(0.f, 0.f);
    return;
  }
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) lab_set_error(LAB_ERR_PAGE_RANGE);
    return;
  }
  const int blocks = (rows + BLK - 1) / BLK;
  if (blocks == 0) return;
  const float* records = p.rec + ((size_t)h * n_records + first_block(row0, req)) * BREC;
  // Chunks come by bulk copies, which cost the walk one thread's instruction (copies of 16 bytes by all threads held its
  // own loads up: 1,400 of a chunk's 6,500 cycles).
  uint64_t* here = reinterpret_cast<uint64_t*>(blocks_smem + 2 * BCHUNK * BREC);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(here + 2);
  if (tid == 0) {
    mbar_init(&here[0], 1), mbar_init(&here[1], 1);
    *abort_flag = 0;
    mbar_init_fence();
  }
  __syncthreads();
  int sent = 0;                   // chunks whose copies have set out (thread 0)
  auto fetch = [&](int b0) {      // one thread; a chunk, where there is one
    if (b0 >= blocks) return;
    ++sent;
    const uint32_t bytes = min(BCHUNK, blocks - b0) * BREC * 4;
    uint64_t* bar = &here[b0 / BCHUNK % 2];
    mbar_expect_tx(bar, bytes);
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(blocks_smem + b0 / BCHUNK % 2 * BCHUNK * BREC)),
                 "l"(records + (size_t)b0 * BREC), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
  };
  // A chunk is here and nobody reads the one before it any more; or the wait ran out (the error word says so): the whole block
  // then goes no further than the block at hand.
  auto landed = [&](int b0) {
    mbar_wait(&here[b0 / BCHUNK % 2], b0 / BCHUNK / 2 & 1, abort_flag);
    __syncthreads();
    return *abort_flag == 0;
  };
  if (tid == 0) fetch(0), fetch(BCHUNK);
  float* S_g = p.state + ((size_t)slot * p.heads + h) * D * D + (size_t)(g * SLB) * D + j;
  f32x2 S[NCOL][SLB / 2];
#pragma unroll
  for (int i = 0; i < SLB / 2; ++i) {
    const float2 lo = *reinterpret_cast<const float2*>(S_g + (size_t)(2 * i) * D);
    const float2 hi = *reinterpret_cast<const float2*>(S_g + (size_t)(2 * i + 1) * D);
    S[0][i] = pair_of(lo.x, hi.x), S[1][i] = pair_of(lo.y, hi.y);
  }
  float* out = p.out + (size_t)row0 * p.heads * D + h * D + j;
  bool alive = landed(0);
  const int o_row = g % BLK;      // the token whose output this thread forms (threads g < BLK write)
  // vectors of the block at hand; as soon as one is used up its place takes the next block's
  f32x2 dots[B_DOTS][SLB / 2], keys[BLK][SLB / 2], gone_by[BLK][SLB / 2], decay[SLB / 2];
  const float* share = blocks_smem + g * SLBP;
#pragma unroll
  for (int i = 0; i < B_DOTS; ++i) load_share(dots[i], share, i);
#pragma unroll
  for (int i = 0; i < BLK; ++i) load_share(keys[i], share, B_KEYS + i), load_share(gone_by[i], share, B_GONE + i);
  load_share(decay, share, B_DECAY);
  for (int b = 0; b < blocks && alive; ++b) {
    const float* rec = blocks_smem + (b / BCHUNK % 2 * BCHUNK + b % BCHUNK) * BREC;
    float v[NCOL][BLK], uk[2 * N_PAIR];
#pragma unroll
    for (int i = 0; i < BLK; ++i) {
      const float2 vv = *reinterpret_cast<const float2*>(rec + AT_V + i * D + j);
      v[0][i] = vv.x, v[1][i] = vv.y;
    }
#pragma unroll
    for (int i = 0; i < 2 * N_PAIR / 4; ++i) {
      const float4 f = *reinterpret_cast<const float4*>(rec + AT_C + 4 * i);
      uk[4 * i] = f.x, uk[4 * i + 1] = f.y, uk[4 * i + 2] = f.z, uk[4 * i + 3] = f.w;
    }
    const float4 rk = *reinterpret_cast<const float4*>(rec + AT_C + C_RK + BLK * o_row);
    const float4 ra = *reinterpret_cast<const float4*>(rec + AT_C + C_RA + BLK * o_row);
    f32x2 s2[NCOL][B_DOTS];
#pragma unroll
    for (int c = 0; c < NCOL; ++c)
#pragma unroll
      for (int i = 0; i < B_DOTS; ++i) s2[c][i] = mul2(dots[i][0], S[c][0]);
#pragma unroll
    for (int q = 1; q < SLB / 2; ++q)
#pragma unroll
      for (int c = 0; c < NCOL; ++c)
#pragma unroll
        for (int i = 0; i < B_DOTS; ++i) fma_pair(s2[c][i], dots[i][q], S[c][q]);
    // the next block (after the last one this one again, for nothing), in the other buffer where a chunk ends
    const int nb = min(b + 1, blocks - 1);
    if (nb % BCHUNK == 0 && nb > b) {
      alive = landed(nb);
      if (tid == 0) fetch(nb + BCHUNK);
    }
    share = blocks_smem + (nb / BCHUNK % 2 * BCHUNK + nb % BCHUNK) * BREC + g * SLBP;
    float t[NCOL][B_DOTS], mine[NCOL];
#pragma unroll
    for (int c = 0; c < NCOL; ++c)
#pragma unroll
      for (int i = 0; i < B_DOTS; ++i) t[c][i] = low_of(s2[c][i]) + high_of(s2[c][i]);
    // every thread of a column needs what is removed; a token's output is formed by one (its sums are passed on alone)
#pragma unroll
    for (int o = 1; o < GB; o <<= 1)
#pragma unroll
      for (int c = 0; c < NCOL; ++c)
#pragma unroll
        for (int i = 0; i < BLK; ++i) t[c][i] += __shfl_xor_sync(0xffffffffu, t[c][i], o);
#pragma unroll
    for (int i = 0; i < B_DOTS; ++i) load_share(dots[i], share, i);
    const bool hi2 = g & 2, hi1 = g & 1;
#pragma unroll
    for (int c = 0; c < NCOL; ++c) {
      const float a0 = (hi2 ? t[c][6] : t[c][4]) + __shfl_xor_sync(0xffffffffu, hi2 ? t[c][4] : t[c][6], 2);
      const float a1 = (hi2 ? t[c][7] : t[c][5]) + __shfl_xor_sync(0xffffffffu, hi2 ? t[c][5] : t[c][7], 2);
      mine[c] = (hi1 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, hi1 ? a0 : a1, 1);
#pragma unroll
      for (int o = 4; o < GB; o <<= 1) mine[c] += __shfl_xor_sync(0xffffffffu, mine[c], o);
    }
    // what does not wait for the sums
#pragma unroll
    for (int c = 0; c < NCOL; ++c)
#pragma unroll
      for (int q = 0; q < SLB / 2; ++q) {
        S[c][q] = mul2(decay[q], S[c][q]);
#pragma unroll
        for (int i = 0; i < BLK; ++i) fma_pair(S[c][q], keys[i][q], pair_of(v[c][i], v[c][i]));
      }
    load_share(decay, share, B_DECAY);
#pragma unroll
    for (int i = 0; i < BLK; ++i) load_share(keys[i], share, B_KEYS + i);
    float result[NCOL];
#pragma unroll
    for (int c = 0; c < NCOL; ++c) {
      float gone[BLK];
      int pair = 0;
#pragma unroll
      for (int i = 0; i < BLK; ++i) {
        float known = 0.f;
#pragma unroll
        for (int jj = 0; jj < i; ++jj) known = fmaf(uk[C_UK + pair + jj], v[c][jj], known);
        gone[i] = t[c][i] + known;
#pragma unroll
        for (int jj = 0; jj < i; ++jj) gone[i] = fmaf(uk[C_UA + pair + jj], gone[jj], gone[i]);
        pair += i;
      }
#pragma unroll
      for (int q = 0; q < SLB / 2; ++q)
#pragma unroll
        for (int i = 0; i < BLK; ++i) fma_pair(S[c][q], gone_by[i][q], pair_of(gone[i], gone[i]));
      // (a later token's numbers stay out: zero times an infinity would be none)
      auto upto = [&](int jj, float f) { return jj <= o_row ? f : 0.f; };
      const float held = fmaf(rk.w, upto(3, v[c][3]), fmaf(rk.z, upto(2, v[c][2]), fmaf(rk.y, upto(1, v[c][1]), rk.x * v[c][0])));
      const float lost = fmaf(ra.w, upto(3, gone[3]), fmaf(ra.z, upto(2, gone[2]), fmaf(ra.y, upto(1, gone[1]), ra.x * gone[0])));
      result[c] = mine[c] + (held + lost);
    }
#pragma unroll
    for (int i = 0; i < BLK; ++i) load_share(gone_by[i], share, B_GONE + i);
    const int row = b * BLK + o_row;
    if (g < BLK && row < rows) *reinterpret_cast<float2*>(out + (size_t)row * p.heads * D) = make_float2(result[0], result[1]);
  }
  if (!alive) {      // copies in flight land before the block's shared memory goes away
    if (tid == 0)
      for (int c = max(0, sent - 2); c < sent; ++c) {
        const uint64_t t0 = global_timer_ns();
        while (!mbar_try_wait(&here[c % 2], c / 2 & 1) && global_timer_ns() - t0 < 100000000ull) {
        }
      }
    return;
  }
  pdl_trigger();      // (not earlier: the next kernel's blocks would settle beside this one's and slow them down)
  if (p.write) {
#pragma unroll
    for (int i = 0; i < SLB / 2; ++i) {
      *reinterpret_cast<float2*>(S_g + (size_t)(2 * i) * D) = make_float2(low_of(S[0][i]), low_of(S[1][i]));
      *reinterpret_cast<float2*>(S_g + (size_t)(2 * i + 1) * D) = make_float2(high_of(S[0][i]), high_of(S[1][i]));
    }
  }
}

// Each head's raw output divided by its root mean square, times a plain weight and sigmoid(gate),
// rounded to T: one CTA per token, a warp per head at a time.
template <typename T>
__global__ void __launch_bounds__(256) delta_finish_kernel(T* __restrict__ out, const float* __restrict__ raw,
                                                           const float* __restrict__ gate, int ld_gate,
                                                           const T* __restrict__ norm_w, int heads, float eps) {
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int h = blockIdx.y * 8 + warp; h < heads; h += 8 * gridDim.y) {
    const float* o = raw + ((size_t)t * heads + h) * D;
    float ss = 0.f;
    for (int i = lane; i < D; i += 32) ss += o[i] * o[i];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)D + eps);
    for (int i = lane; i < D; i += 32)
      out[((size_t)t * heads + h) * D + i] =
          from_f32<T>(o[i] * inv * to_f32(norm_w[h * D + i]) * sigmoidf_(gate[(size_t)t * ld_gate + h * D + i]));
  }
}

// out (T) [tokens, n] = tanh(x [tokens, ld]) for the low-rank middle of the decay's projection
template <typename T>
__global__ void __launch_bounds__(256) tanh_cast_kernel(T* __restrict__ out, const float* __restrict__ x, long long tokens,
                                                        int n, int ld) {
  pdl_trigger();
  pdl_wait();
  const long long total = tokens * n;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256)
    out[i] = from_f32<T>(tanhf(x[(i / n) * ld + (i % n)]));
}

}  // namespace

LAB_EXPORT int lab_delta_rule_head_dim() { return D; }

namespace {
// Raw outputs lie first in the scratch, the records behind them on a boundary of 16 bytes.
inline float* records_of(float* scratch, int tokens, int heads) { return scratch + ((size_t)tokens * heads * D + 3) / 4 * 4; }

template <typename T>
int launch_blocks(const DeltaParams& p, const float* r, const float* k, const float* v, const float* a, int ld, const float* d,
                  int ld_d, const T* d_bias, const T* a_bias, int requests, float decay_rate, cudaStream_t stream) {
  static LabShared granted;
  cudaError_t e = lab_allow_shared(granted, (const void*)delta_blocks_kernel, BSMEM);
  if (e != cudaSuccess) return (int)e;
  const int n_records = p.tokens / BLK + requests;
  e = lab_launch(delta_prepare_blocks_kernel<T>, dim3(n_records, (p.heads + 7) / 8), dim3(256), 0, stream, (float*)p.rec,
                 n_records, r, k, v, a, ld, d, ld_d, d_bias, a_bias, p.q_start, requests, p.heads, decay_rate);
  if (e != cudaSuccess) return (int)e;
  return (int)lab_launch(delta_blocks_kernel, dim3(p.heads, requests, D / BCOLS), dim3(BTHREADS), BSMEM, stream, p, n_records);
}

template <typename T>
int launch_delta_rule(DeltaParams p, void* out, const float* r, const float* k, const float* v, const float* g, const float* a,
                      int ld, const float* d, int ld_d, const T* d_bias, const T* a_bias, const T* norm_w, int requests,
                      int blocks, float eps, float decay_rate, cudaStream_t stream) {
  // the kernels that are parallel over tokens: a warp per (token, head); with few tokens the heads spread over CTAs as well
  const dim3 per_token(p.tokens, p.tokens >= 512 ? 1 : (p.heads + 7) / 8);
  int e = (int)cudaErrorInvalidValue;
  if (blocks != 0) {
    if constexpr (BLOCKS_BUILT && !std::is_same_v<T, float>)
      e = launch_blocks<T>(p, r, k, v, a, ld, d, ld_d, d_bias, a_bias, requests, decay_rate, stream);
  } else {
    static LabShared granted;
    e = (int)lab_allow_shared(granted, (const void*)delta_rule_kernel<T>, sizeof(DeltaShared));
    if (e != 0) return e;
    e = (int)lab_launch(delta_prepare_kernel<T>, per_token, dim3(256), 0, stream, (float*)p.rec, p.tokens, r, k, v, a, ld, d, ld_d,
                        d_bias, a_bias, p.heads, decay_rate);
    if (e != 0) return e;
    e = (int)lab_launch(delta_rule_kernel<T>, dim3(p.heads, requests, NS), dim3(NT), sizeof(DeltaShared), stream, p);
  }
  if (e != 0) return e;
  return (int)lab_launch(delta_finish_kernel<T>, per_token, dim3(256), 0, stream, (T*)out, (const float*)p.out, g, ld, norm_w,
                         p.heads, eps);
}
}  // namespace

// Whether the walk by blocks of four tokens is built for this head size.
LAB_EXPORT int lab_delta_rule_blocks() { return BLOCKS_BUILT; }

// Floats of scratch: the heads' raw outputs and the records.  blocks: as lab_delta_rule takes it.
LAB_EXPORT long long lab_delta_rule_scratch(int tokens, int heads, int requests, int blocks) {
  const long long records = blocks != 0 ? ((long long)tokens / BLK + requests) * BREC : (long long)tokens * REC;
  return (long long)tokens * heads * D + 4 + heads * records;
}

// blocks: 0, a token at a time; 1 (16-bit storage, where lab_delta_rule_blocks), four at a time.
LAB_EXPORT int lab_delta_rule(void* out, float* scratch, const float* r, const float* k, const float* v,
                              const float* g, const float* a, int ld, const float* d, int ld_d, const void* d_bias,
                              const void* a_bias, const void* norm_w, float* state, const int* q_start,
                              const int* state_slot, int tokens, int n_requests, int heads, int n_slots, int write,
                              int blocks, float eps, float decay_rate, int dtype, cudaStream_t stream) {
  if (n_requests <= 0 || heads <= 0 || tokens <= 0) return 0;
  DeltaParams p;
  p.out = scratch; p.rec = records_of(scratch, tokens, heads); p.tokens = tokens; p.state = state; p.q_start = q_start;
  p.state_slot = state_slot; p.heads = heads; p.n_slots = n_slots; p.write = write;
  if (dtype == LAB_F32)
    return launch_delta_rule<float>(p, out, r, k, v, g, a, ld, d, ld_d, (const float*)d_bias, (const float*)a_bias,
                                    (const float*)norm_w, n_requests, blocks, eps, decay_rate, stream);
  return launch_delta_rule<__nv_bfloat16>(p, out, r, k, v, g, a, ld, d, ld_d, (const __nv_bfloat16*)d_bias,
                                          (const __nv_bfloat16*)a_bias, (const __nv_bfloat16*)norm_w, n_requests, blocks, eps,
                                          decay_rate, stream);
}

LAB_EXPORT int lab_tanh_cast(void* out, const float* x, long long tokens, int n, int ld, int dtype,
                             cudaStream_t stream) {
  const long long total = tokens * n;
  if (total <= 0) return 0;
  const int blocks = (int)((total + 255) / 256 < 148 * 8 ? (total + 255) / 256 : 148 * 8);
  if (dtype == LAB_F32)
    lab_launch(tanh_cast_kernel<float>, dim3(blocks), dim3(256), 0, stream, (float*)out, x, tokens, n, ld);
  else
    lab_launch(tanh_cast_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, (__nv_bfloat16*)out, x, tokens, n,
               ld);
  LAB_LAUNCH_CHECK();
}
