// 32-bit matrix product on the tensor cores: every operand is cut into three bfloat16 numbers, whose products the tensor cores
// form exactly.
//
//   out[m, n] = sum_k x[m, k] * w[n, k]  (+ bias[n]; activation)      or gated, as in gemm_plain.cu; w is [out, in]
//
// A number's first 8 bits, the first 8 of what is left and the rest, 8 at most, make it up exactly: x = x1 + x2 + x3, |x2| <
// 2^-7 |x|, |x3| < 2^-15 |x|.  A product is w1 x1 + (w1 x2 + w2 x1 + w2 x2 + w1 x3 + w3 x1 + w2 x3 + w3 x2); what is dropped,
// w3 x3, is below 2^-30 of it.  Both operands enter times 2^24: the tensor cores take numbers below the smallest normal one for
// zero, and so neither a part of an operand nor a product that counts is below it.  The sum over k: the tensor cores add up
// chunks of 32 k's, w1 x1 and the small products apart, in steps of 16 k's at which a sum loses what lies below its last bit;
// the chunks go one after the other into a sum kept in registers, rounded to nearest.  K is cut into F32_PARTS parts of whole
// chunks, which are added pairwise, as a tree.  None of this depends on the rows that come together or on the tile, so neither
// does any bit of the output.  A row of x whose one entry is a power of two gives w's column back, bit for bit.  2-norm of the
// error (multiply-adds in brackets, in the order of gemm_plain.cu): normal operands, 896 k's 7.9e-8 (2.0e-7), 4,864 1.1e-7
// (4.5e-7); operands from 0.5 to 1.5 3.7e-8 (6.0e-8) and 5.0e-8 (1.4e-7); over eight decades 9.6e-8 (1.4e-7) and 1.2e-7
// (3.0e-7); operands of 1e-38, or 1e-40 by 1e18, likewise.
//
// What bounds it: the products' issue and the chain of hand-overs a chunk passes (brought, cut, multiplied, summed), 850 to
// 1,300 cycles a chunk whatever the tile; 512 of them are products where a tile has 64 rows.  Three products instead of eight
// would save 15 %, a third part that is neither formed nor stored 4 to 10 %; deeper rings, more sums in tensor memory, two
// chunks at a time and two CTAs a multiprocessor did not shorten the chain.  Sums of parts that wait for their neighbour's lie
// in local memory in the larger tiles, touched once a part.  Measured on a B200, weights from memory, against tiles of 64 x 64
// by fused multiply-adds, which reach half of the units' rate (us): 517 x 4,864 x 896 gated 146 (266), 517 x 896 x 4,864 56
// (157), 517 x 1,152 x 896 31 (43), 517 x 896 x 896 18 (34), 100 x 896 x 4,864 18 (75), 8 x 896 x 4,864 13 (17); few rows with
// short K are slower, 8 x 1,152 x 896 6.1 (5.1), 8 x 4,864 x 896 gated 18.5 (13.2), 1 x 4,864 x 896 gated 18 (9.3), rows on no 16
// bytes 1 x 4,864 x 898 gated 36 (31), but a row's bits may not depend on how many come with it.
//
// A result that is no finite number, or beyond 2^79, is formed again by fused multiply-adds, in gemm_plain.cu's order: an
// infinite operand, or a sum that outgrows 32 bits times 2^48, leaves differences of infinities behind.
#pragma once
#include "tcgen05.cuh"

namespace {
constexpr int F32_PARTS = 8;        // parts of K, at most a cluster of CTAs
constexpr int F32_CHUNK = 32;       // k's of a chunk: rows of 128 bytes, one swizzled row
constexpr int F32_FEATURES = 128;   // rows of w a tile holds (gated: 64 gate and 64 up)
constexpr int F32_GROUP = 128;      // threads of a group that splits operands
constexpr int F32_THREADS = 128 + 2 * F32_GROUP + 64;      // sums; two such groups; issue; loads

// Whether this lane issues (one of a converged warp).  Asked once for a run of products: an election in each took a third of
// their issue.
__device__ __forceinline__ uint32_t elected() {
  uint32_t e;
  asm volatile("{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\tselp.u32 %0, 1, 0, e;\n\t}" : "=r"(e));
  return e;
}
// D[tmem] (+)= A[tmem] * B[smem]^T by the lane that `issues`, as umma_bf16_tmem_a.
template <bool ADD>
__device__ __forceinline__ void f32_mma(uint32_t issues, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, e;\n\t"
      "setp.ne.b32 e, %4, 0;\n\t"
      "setp.ne.b32 p, %5, 0;\n\t"
      "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%6, %6, %6, %6}, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(issues), "n"(ADD ? 1 : 0), "r"(0u)
      : "memory");
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
// The first 8 bits of each of two numbers side by side; the two become what is left of them, exactly.
__device__ __forceinline__ uint32_t heads_of(unsigned long long& pair) {
  const uint32_t a = (uint32_t)pair, b = (uint32_t)(pair >> 32);
  const unsigned long long heads = (unsigned long long)(b & 0xffff0000u) << 32 | (a & 0xffff0000u);
  pair = fma2(heads, pair_of(-1.f, -1.f), pair);
  return __byte_perm(a, b, 0x7632);
}
constexpr float F32_SCALE = 16777216.f;      // 2^24: what both operands enter the product times

struct F32Params {
  float* out;
  const float *x, *w, *bias;
  int M, N, K, ldx, ldo;
  int act;              // plain: 0, or the activation's code; gated: the gate's
  float gate_limit;
  int chunks, part_chunks;
  unsigned m_tiles, tiles;
};

// 4 bytes, zeros where `has` is false, from global to shared memory without a register in between.
__device__ __forceinline__ void f32_copy4(uint32_t dst, const void* src, bool has) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(has ? 4 : 0) : "memory");
}

template <int NT> struct F32Tile {      // NT rows of x
  static constexpr int A_BYTES = F32_FEATURES * 128, B_BYTES = NT * 128;
  static constexpr int STAGE = A_BYTES + 2 * B_BYTES;          // w's rows as they are; x1 beside x2, x3 in half a row
  static constexpr int STAGES = 220 * 1024 / STAGE;            // 11, 9 or 6
  static constexpr int SMEM = STAGES * STAGE + 1024 + 512;
  static constexpr int SUMS = 2 * NT;                          // columns of a chunk's sums: w1 x1, the small products
  // chunks in tensor memory: their sums, and behind those their w1, w2, w3 (two k's a column)
  static constexpr int SUM_BUFS = NT <= 32 ? 4 : 3, W_BUFS = NT <= 32 ? 4 : 2;
  static constexpr int W_AT = SUM_BUFS * SUMS, W_COLUMNS = 3 * F32_CHUNK / 2;
  static constexpr int TMEM = 512;
  static_assert(W_AT + W_BUFS * W_COLUMNS <= TMEM, "tensor memory");
  static_assert(NT * F32_FEATURES * 4 <= STAGES * STAGE, "the parts' sums lie in the stages");
  static_assert((3 * STAGES + 2 * SUM_BUFS) * 8 + 8 <= 512, "the barriers outgrow their 512 bytes");
};

// A CTA takes 128 rows of w by NT of x: features lie along the lanes of tensor memory, so a warp stores 128 bytes of a
// row.  One warp brings both operands' chunks (TMA); two groups of four warps take every other chunk and split it, w's rows,
// a thread a row, into tensor memory, x's in place; one warp issues the products; four add up the chunks' sums and finish.
// SPREAD CTAs (1 to F32_PARTS), a cluster, share the parts of K and add their sums through one another's shared memory.
// A CTA without a cluster walks several tiles, the sums of one finished beside the products of the next.
// VEC: rows lie on 16-byte boundaries, as TMA wants them; else the groups copy their chunk themselves, element by element.
template <bool GATED, int NT, bool VEC, int SPREAD>
__global__ void __launch_bounds__(F32_THREADS, 1) gemm_f32_kernel(const __grid_constant__ CUtensorMap map_w,
                                                                  const __grid_constant__ CUtensorMap map_x, F32Params p) {
  using Tile = F32Tile<NT>;
  constexpr int STAGES = Tile::STAGES;
  extern __shared__ uint8_t f32_raw[];
  uint8_t* tiles = (uint8_t*)(((uintptr_t)f32_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* raw = (uint64_t*)(tiles + STAGES * Tile::STAGE);      // a chunk is here, it is split, it has been multiplied
  uint64_t* full = raw + STAGES;
  uint64_t* empty = full + STAGES;
  constexpr int SUM_BUFS = Tile::SUM_BUFS;
  uint64_t* sum_full = empty + STAGES;      // [SUM_BUFS]
  uint64_t* sum_empty = sum_full + SUM_BUFS;
  uint32_t* tmem_slot = (uint32_t*)(sum_empty + SUM_BUFS);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // tiles of one block of features lie side by side: they read the same rows of w
  auto row_of_tile = [&](unsigned tile) { return (int)(tile % p.m_tiles) * NT; };
  auto feature_of_tile = [&](unsigned tile) { return (int)(tile / p.m_tiles) * (GATED ? F32_FEATURES / 2 : F32_FEATURES); };
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&raw[s], 1);
      mbar_init(&full[s], F32_GROUP / 32);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < SUM_BUFS; ++b) {
      mbar_init(&sum_full[b], 1);
      mbar_init(&sum_empty[b], 4);
    }
    *abort_flag = 0;
    mbar_init_fence();
  }
  if (warp == 0) tmem_alloc(tmem_slot, Tile::TMEM);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_wait();

  constexpr int OWN = F32_PARTS / SPREAD;      // parts of this CTA
  const int first_part = (int)blockIdx.y * OWN, last_part = first_part + OWN;
  const int c_begin = min(p.chunks, first_part * p.part_chunks);
  const int n_chunks = min(p.chunks, last_part * p.part_chunks) - c_begin;
  const int own_tiles = blockIdx.x < p.tiles ? (int)((p.tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
  // What follows the product, for columns m.. of this lane (warps 0..3, every lane): lane r holds feature n0 + r, of a gated
  // tile 16 gate rows and then their up rows in each warp.
  const int r = (warp & 3) * 32 + lane;
  auto finish = [&](auto& v, int n0, int m) {
    constexpr int COUNT = sizeof(v) / sizeof(float);
    const int n = n0 + (GATED ? (r >> 5) * 16 + (r & 15) : r);
    const float bias = !GATED && p.bias != nullptr && n < p.N ? p.bias[n] : 0.f;
    unsigned long long again = 0ull;
#pragma unroll
    for (int j = 0; j < COUNT; ++j) {
      v[j] *= 1.f / (F32_SCALE * F32_SCALE);
      if (!(fabsf(v[j]) <= 3.402823466e38f) && m + j < p.M && n < p.N) again |= 1ull << j;
    }
    while (again != 0ull) {
      const int j = __ffsll((long long)again) - 1;
      again &= again - 1;
      const float *a = p.w + (size_t)(GATED && (r & 16) ? p.N + n : n) * p.K, *b = p.x + (size_t)(m + j) * p.ldx;
      float s[8] = {};
#pragma unroll 1
      for (int k = 0; k < p.K; ++k) {
        const int q = k / 16 % 4 * 2 + k % 2;
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = i == q ? fmaf(__ldg(a + k), __ldg(b + k), s[i]) : s[i];
      }
      const float sum = (s[0] + s[1] + (s[2] + s[3])) + (s[4] + s[5] + (s[6] + s[7]));
#pragma unroll
      for (int i = 0; i < COUNT; ++i) v[i] = i == j ? sum : v[i];
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < COUNT; ++j) {
      if (GATED) {      // two columns at a time: a lane of gates finishes the first, its partner the second
        if (j % 2 != 0) continue;
        const bool up = (lane & 16) != 0;
        const float theirs = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + 1], 16);
        const float g = up ? theirs : v[j], u = up ? v[j + 1] : theirs;
        const int mine = m + j + (up ? 1 : 0);
        if (mine < p.M && n < p.N) p.out[(size_t)mine * p.ldo + n] = gate_pair(g, u, p.act, p.gate_limit);
      } else if (m + j < p.M && n < p.N) {
        const float t = v[j] + bias;
        p.out[(size_t)(m + j) * p.ldo + n] = p.act ? lab_act(t, p.act) : t;
      }
    }
  };

  float acc[NT];      // (warps 0..3) the sums of this thread's lane
  if (warp < 4) {
    const uint32_t mine = tmem + ((uint32_t)(warp * 32) << 16);
    float waiting[OWN > 4 ? 3 : OWN > 2 ? 2 : 1][NT];      // sums of whole subtrees that wait for their neighbour's
    int it = 0;
    bool ok = true;
#pragma unroll 1
    for (unsigned tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
#pragma unroll 1
      for (int part = 0; part < OWN && ok; ++part) {
        const int b = min(p.chunks, (first_part + part) * p.part_chunks), e = min(p.chunks, b + p.part_chunks);
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[j] = 0.f;
        for (int c = b; c < e; ++c, ++it) {
          const int buf = it % SUM_BUFS;
          ok = __all_sync(0xffffffffu, mbar_wait(&sum_full[buf], (it / SUM_BUFS) & 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int g = 0; g < NT; g += 16) {
            uint32_t large[16], small[16];
            tmem_ld16_issue(mine + buf * Tile::SUMS + g, large);
            tmem_ld16_issue(mine + buf * Tile::SUMS + NT + g, small);
            tmem_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[g + j] += __uint_as_float(large[j]) + __uint_as_float(small[j]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sum_empty[buf]);
        }
        int level = 0;
        for (int rest = part; rest & 1; rest >>= 1, ++level) {
#pragma unroll
          for (int j = 0; j < NT; ++j) acc[j] = waiting[level][j] + acc[j];
        }
        if (part + 1 < OWN) {
#pragma unroll
          for (int j = 0; j < NT; ++j) waiting[level][j] = acc[j];
        }
      }
      if (SPREAD == 1 && ok) finish(acc, feature_of_tile(tile), row_of_tile(tile));
    }
  } else if (warp < 4 + 2 * F32_GROUP / 32) {
    // a thread's units of x: 16 bytes of every 16th row
    constexpr int STEP = F32_GROUP / 8, NB = NT / STEP;
    const int group = (warp - 4) / (F32_GROUP / 32), t = tid % F32_GROUP, unit = t & 7, row0 = t >> 3;
    const uint32_t at = row0 * 128 + ((unit ^ (row0 & 7)) << 4);      // (STEP rows on: the same place in the swizzle)
    constexpr int W_BUFS = Tile::W_BUFS;
    // where a unit's parts go: 8 bytes of x1, of x2 64 bytes on in the row, of x3 in the second array
    const uint32_t at1 = row0 * 128 + (((unit >> 1) ^ (row0 & 7)) << 4) + (unit & 1) * 8;
    const uint32_t at2 = row0 * 128 + (((4 + (unit >> 1)) ^ (row0 & 7)) << 4) + (unit & 1) * 8;
    const uint32_t w_tmem = tmem + ((uint32_t)((warp & 3) * 32) << 16) + Tile::W_AT;
    // where row t of tensor memory lies in a stage (gated: all gate rows come first)
    const int w_row = GATED ? (t & 16) * 4 + (t >> 5) * 16 + (t & 15) : t;
    auto multiplied = [&](int c) {
      return c < 0 || __all_sync(0xffffffffu, mbar_wait(&empty[c % STAGES], (c / STAGES) & 1, abort_flag));
    };
    int first = 0;      // the tile's first chunk, counted over all of this CTA's
    bool ok = true;
    for (unsigned tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x, first += n_chunks) {
      const int m0 = row_of_tile(tile), n0 = feature_of_tile(tile);
      for (int c = first + ((first ^ group) & 1); c < first + n_chunks; c += 2) {
        ok = false;
        uint8_t *stage = tiles + c % STAGES * Tile::STAGE, *x_stage = stage + Tile::A_BYTES;
        if constexpr (VEC) {
          if (!__all_sync(0xffffffffu, mbar_wait(&raw[c % STAGES], (c / STAGES) & 1, abort_flag))) break;
        } else {
          if (!multiplied(c - STAGES)) break;
          const int k = (c_begin + c - first) * F32_CHUNK + unit * 4;
          for (int i = 0; i < F32_FEATURES / STEP + NB; ++i) {
            const bool of_x = i >= F32_FEATURES / STEP;
            const int r = row0 + STEP * (of_x ? i - F32_FEATURES / STEP : i);
            const int f = n0 + (GATED ? r % 64 : r);
            const bool live = of_x ? m0 + r < p.M : f < p.N;
            const float* row = of_x ? p.x + (size_t)(m0 + r) * p.ldx : p.w + (size_t)(GATED && r >= 64 ? p.N + f : f) * p.K;
            const uint32_t to = smem_u32(of_x ? x_stage : stage) + (r - row0) * 128 + at;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const bool has = live && k + e < p.K;
              f32_copy4(to + 4 * e, has ? row + k + e : p.x, has);
            }
          }
          asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
          if (group == 0) asm volatile("bar.sync 1, %0;" ::"n"(F32_GROUP) : "memory");      // the group's copies are here
          else asm volatile("bar.sync 2, %0;" ::"n"(F32_GROUP) : "memory");
        }
        unsigned long long v[F32_CHUNK / 2];      // row t of w
#pragma unroll
        for (int u = 0; u < F32_CHUNK / 4; ++u) {
          const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(stage + w_row * 128 + ((u ^ (w_row & 7)) << 4));
          v[2 * u] = q.x, v[2 * u + 1] = q.y;
        }
        float4 x[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) x[i] = *reinterpret_cast<const float4*>(x_stage + i * STEP * 128 + at);
        __syncwarp();      // a row's parts take the row's place; its eight units are this warp's
        uint32_t w12[F32_CHUNK], w3[F32_CHUNK / 2];
#pragma unroll
        for (int e = 0; e < F32_CHUNK / 2; ++e) {
          v[e] = mul2(v[e], pair_of(F32_SCALE, F32_SCALE));
          w12[e] = heads_of(v[e]), w12[F32_CHUNK / 2 + e] = heads_of(v[e]), w3[e] = heads_of(v[e]);
        }
        if (!multiplied(c - W_BUFS)) break;      // its place in tensor memory is free
        tc_fence_after();
        const uint32_t to = w_tmem + c % W_BUFS * Tile::W_COLUMNS;
        tmem_st32(to, w12);
        tmem_st16(to + F32_CHUNK, w3);
#pragma unroll
        for (int i = 0; i < NB; ++i) {
          uint8_t* into = x_stage + i * STEP * 128;
          unsigned long long lo = pair_of(x[i].x * F32_SCALE, x[i].y * F32_SCALE), hi = pair_of(x[i].z * F32_SCALE, x[i].w * F32_SCALE);
          uint2 part[3];
#pragma unroll
          for (int q = 0; q < 3; ++q) part[q].x = heads_of(lo), part[q].y = heads_of(hi);
          *reinterpret_cast<uint2*>(into + at1) = part[0];
          *reinterpret_cast<uint2*>(into + at2) = part[1];
          *reinterpret_cast<uint2*>(into + Tile::B_BYTES + at1) = part[2];
        }
        proxy_fence();
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[c % STAGES]);
        ok = true;
      }
    }
  } else if (warp == 4 + 2 * F32_GROUP / 32) {
    auto wait_all = [&](uint64_t* bar, uint32_t parity) {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
    };
    constexpr uint32_t idesc = umma_instr_desc(F32_FEATURES, NT);
    // (places and phases are counted on: divisions by the numbers of stages and buffers would be a third of the loop)
    int s = 0, buf = 0, w_buf = 0;
    uint32_t phase = 0, sum_phase = 1;
    const int all = own_tiles * n_chunks;
    const uint32_t issues = elected();
    for (int c = 0; c < all; ++c) {
      if (!wait_all(&sum_empty[buf], sum_phase) || !wait_all(&full[s], phase)) break;
      tc_fence_after();
      const uint32_t large = tmem + buf * Tile::SUMS, small = large + NT, w = tmem + Tile::W_AT + w_buf * Tile::W_COLUMNS;
      const uint64_t x1 = smem_desc_sw128(smem_u32(tiles + s * Tile::STAGE + Tile::A_BYTES));
      const uint64_t x[3] = {x1, x1 + 4, x1 + Tile::B_BYTES / 16};      // (x2 lies 64 bytes on in x1's rows)
      // w1 x1 of both halves of the chunk; the small ones
      constexpr int HALF = F32_CHUNK / 2;
      f32_mma<false>(issues, large, w, x[0], idesc);
      f32_mma<true>(issues, large, w + 8, x[0] + 2, idesc);
      f32_mma<false>(issues, small, w, x[1], idesc);
#pragma unroll
      for (int q = 1; q < 8; ++q)      // w1 x2, w1 x3, w2 x1, w2 x2, w2 x3, w3 x1, w3 x2: 16 k's are 8 columns of w, 32 bytes of x
#pragma unroll
        for (int k = q == 1 ? 1 : 0; k < 2; ++k) f32_mma<true>(issues, small, w + HALF * (q / 3) + 8 * k, x[q % 3] + 2 * k, idesc);
      umma_commit(&empty[s]);
      umma_commit(&sum_full[buf]);
      if (++s == STAGES) s = 0, phase ^= 1;
      if (++buf == SUM_BUFS) buf = 0, sum_phase ^= 1;
      if (++w_buf == Tile::W_BUFS) w_buf = 0;
    }
  } else if (VEC && lane == 0) {
    int c = 0;
    bool ok = true;
    for (unsigned tile = blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
      const int m0 = row_of_tile(tile), n0 = feature_of_tile(tile);
      for (int i = 0; i < n_chunks; ++i, ++c) {
        const int s = c % STAGES, k = (c_begin + i) * F32_CHUNK;
        ok = c < STAGES || mbar_wait(&empty[s], (c / STAGES - 1) & 1, abort_flag);
        if (!ok) break;
        mbar_expect_tx(&raw[s], Tile::A_BYTES + Tile::B_BYTES);
        const uint32_t to = smem_u32(tiles + s * Tile::STAGE);
        tma_load_2d(to, &map_w, &raw[s], k, n0);
        if (GATED) tma_load_2d(to + Tile::A_BYTES / 2, &map_w, &raw[s], k, p.N + n0);      // 64 gate rows, then their up rows
        tma_load_2d(to + Tile::A_BYTES, &map_x, &raw[s], k, m0);
      }
    }
    if (*abort_flag) {      // copies in flight land before the CTA's shared memory goes away
      for (int i = c > STAGES ? c - STAGES : 0; i < c; ++i) {
        const uint64_t t0 = global_timer_ns();
        while (!mbar_try_wait(&raw[i % STAGES], (i / STAGES) & 1) && global_timer_ns() - t0 < 100000000ull) {
        }
      }
    }
  }

  // ---- the parts' sums, and the end ----
  if constexpr (SPREAD > 1) {
    // a CTA's sums as [column][lane] in its own shared memory (whose stages have all been read: the last sums waited for
    // that); CTA y finishes NT / SPREAD columns
    float* sums = (float*)tiles;
    if (warp < 4) {
#pragma unroll
      for (int j = 0; j < NT; ++j) sums[j * F32_FEATURES + r] = acc[j];
    }
    tc_fence_before();
    cluster_sync();
    constexpr int EACH = NT / SPREAD;
    static_assert(EACH % 2 == 0, "pairs of columns");
    if (warp < 4 && *abort_flag == 0) {
      const int col = (int)blockIdx.y * EACH;
      const uint32_t at = smem_u32(sums + col * F32_FEATURES + r);
      float v[EACH];
#pragma unroll
      for (int j = 0; j < EACH; ++j) {
        float t[SPREAD];
#pragma unroll
        for (int z = 0; z < SPREAD; ++z) t[z] = ld_cluster_f32(map_to_rank(at + j * F32_FEATURES * 4, z));
#pragma unroll
        for (int o = 1; o < SPREAD; o <<= 1)
#pragma unroll
          for (int z = 0; z < SPREAD; z += 2 * o) t[z] += t[z + o];
        v[j] = t[0];
      }
      finish(v, feature_of_tile(blockIdx.x), row_of_tile(blockIdx.x) + col);
    }
    pdl_trigger();
    cluster_sync();      // the others may still read this CTA's sums
  } else {
    pdl_trigger();
    tc_fence_before();
    __syncthreads();
  }
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, Tile::TMEM);
  }
}

// Map of a row-major matrix of floats with row stride ld, 128-byte swizzle; box = 32 columns by box_rows rows.
inline int f32_map(CUtensorMap* map, const float* base, long long rows, long long cols, long long ld, int box_rows) {
  LabEncodeTiledFn fn = lab_encode_fn();
  if (!fn) return (int)cudaErrorNotSupported;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {(cuuint32_t)F32_CHUNK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <bool GATED, int NT, bool VEC, int SPREAD>
int launch_f32_as(F32Params p, cudaStream_t stream) {
  using Tile = F32Tile<NT>;
  const auto kernel = gemm_f32_kernel<GATED, NT, VEC, SPREAD>;
  static LabShared granted;
  const cudaError_t e = lab_allow_shared(granted, (const void*)kernel, Tile::SMEM);
  if (e != cudaSuccess) return (int)e;
  constexpr int features = GATED ? F32_FEATURES / 2 : F32_FEATURES;
  cudaLaunchConfig_t cfg = {};
  const long long tiles = (long long)((p.N + features - 1) / features) * (p.m_tiles = (unsigned)((p.M + NT - 1) / NT));
  if (tiles > 0x7fffffffll) return (int)cudaErrorInvalidValue;
  p.tiles = (unsigned)tiles;
  cfg.gridDim = dim3((unsigned)(SPREAD > 1 || tiles < lab_sm_count() ? tiles : lab_sm_count()), SPREAD);
  cfg.blockDim = dim3(F32_THREADS);
  cfg.dynamicSmemBytes = Tile::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (g_lab_pdl) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (SPREAD > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = 1, attr[n].val.clusterDim.y = SPREAD, attr[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  CUtensorMap map_w = {}, map_x = {};
  if (VEC) {
    int rc = f32_map(&map_w, p.w, GATED ? 2ll * p.N : p.N, p.K, p.K, GATED ? F32_FEATURES / 2 : F32_FEATURES);
    if (rc == 0) rc = f32_map(&map_x, p.x, p.M, p.K, p.ldx, NT);
    if (rc != 0) return rc;
  }
  return (int)cudaLaunchKernelEx(&cfg, kernel, map_w, map_x, p);
}

// Whether products with these sizes of w go through the tensor cores, by w alone, so that a row's bits depend on nothing that
// comes beside it.  Below 768 k's the fixed cost of a tile leaves little to gain.  Very wide outputs (heads) are asked for few
// rows, which the weights' way from memory bounds there: 1 x 32,768 x 896 36 us here, 22 by multiply-adds, 1 x 151,936 x 896 82
// by multiply-adds.
inline bool f32_on_tensor_cores(int N, int K, bool gated) { return K >= 768 && (gated ? 2ll : 1ll) * N <= 32768; }

// Rows of x a tile holds and CTAs that share the parts of K, by what a launch takes (us): a CTA of 16, 32 or 64 rows 0.47,
// 0.53 or 0.72 a chunk and 3.5 a tile, in clusters 5 and a round more where not all find room at once.
inline void f32_plan(long long M, long long N, bool gated, int chunks, int part_chunks, int& nt, int& spread) {
  const long long sms = lab_sm_count(), blocks = (N + (gated ? 63 : 127)) / (gated ? 64 : 128);
  double best = 0;
  for (int rows = 16; rows <= 64; rows *= 2)
    for (int ctas = 1; ctas <= F32_PARTS; ctas *= 2) {
      const long long room = ctas == 8 ? sms * 7 / 8 : sms;
      const long long rounds = ((M + rows - 1) / rows * blocks * ctas + room - 1) / room;
      const int own = F32_PARTS / ctas * part_chunks < chunks ? F32_PARTS / ctas * part_chunks : chunks;
      const double chunk = rows == 16 ? 0.47 : rows == 32 ? 0.53 : 0.72;
      const double us = ctas == 1 ? rounds * (own * chunk + 3.5) + 4 : rounds * (own * chunk + 5) + 2;
      if (best == 0 || us < best) best = us, nt = rows, spread = ctas;
    }
}

inline int launch_f32(void* out, const void* x, const void* w, const void* bias, int M, int N, int K, int ldx, int ldo,
                      bool gated, int act, float gate_limit, cudaStream_t stream) {
  F32Params p;
  p.out = (float*)out; p.x = (const float*)x; p.w = (const float*)w; p.bias = (const float*)bias;
  p.M = M; p.N = N; p.K = K; p.ldx = ldx; p.ldo = ldo; p.act = act; p.gate_limit = gate_limit;
  p.chunks = (K + F32_CHUNK - 1) / F32_CHUNK;
  p.part_chunks = (p.chunks + F32_PARTS - 1) / F32_PARTS;
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && ldx >= K && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  int nt = 0, spread = 0;
  f32_plan(M, N, gated, p.chunks, p.part_chunks, nt, spread);
#define LAB_F32_AS(GATED_, NT_, VEC_)                                                       \
  return spread == 8   ? launch_f32_as<GATED_, NT_, VEC_, 8>(p, stream)                      \
         : spread == 4 ? launch_f32_as<GATED_, NT_, VEC_, 4>(p, stream)                      \
         : spread == 2 ? launch_f32_as<GATED_, NT_, VEC_, 2>(p, stream)                      \
                       : launch_f32_as<GATED_, NT_, VEC_, 1>(p, stream)
#define LAB_F32_TILE(NT_)                                                                    \
  if (nt == NT_) {                                                                           \
    if (gated && vec) LAB_F32_AS(true, NT_, true);                                           \
    if (gated) LAB_F32_AS(true, NT_, false);                                                 \
    if (vec) LAB_F32_AS(false, NT_, true);                                                   \
    LAB_F32_AS(false, NT_, false);                                                           \
  }
  LAB_F32_TILE(16)
  LAB_F32_TILE(32)
  LAB_F32_TILE(64)
  return (int)cudaErrorInvalidValue;
#undef LAB_F32_AS
#undef LAB_F32_TILE
}
}  // namespace
