// Split-KV decode attention over paged keys and values on the warp-level matrix instructions: one CTA of four
// warps per (sequence, kv head, split), every warp with keys, pipeline and running softmax of its own.
//
// Bound: HBM (every page row is read once).  The scalar form of this kernel (eight lanes per key, dot products and
// P.V on the FMA pipe) was bound by instruction issue instead: 4 query heads per kv head cost 2 x 4 FMA per stored
// element, plus conversions for int8 pages.  Measured for one layer, before -> after:
//   bf16, 64 x 2050 keys, 4 kv heads, group of 4:   105.3 -> 49.8 us (268 MB, 5.4 TB/s; in one split 133 -> 45.5)
//   int8, 200 sequences of 128..2304 keys, 8 kv heads, group of 4:   333 -> 102 us (514 MB, 5.0 TB/s)
//
// Tile: 16 keys.  S^T[16 keys, 8 columns] = K Q^T and O^T[HD, 8 columns] += V^T P^T, so the stored rows are the
// 16-row operands as they lie in memory (V through transposing loads) and the query heads are the eight columns.
// A warp's column fragments keep their lanes from S to O: maximum, sum and rescaling need no exchange but three
// shuffles per tile.  P keeps its 24 bits: three 16-bit pieces that add up to it.  The columns past the heads carry the
// second (and, up to two heads, the third) piece of the same heads, whose scores come from repeated query columns; three and
// four heads take two products, eight take three.  The pieces' sums are added at the end.  The unit cuts its sums off, which
// over a long row of tiles would drift: a tile's products are added up on their own.  Error of the fp32 result against 64 bits
// 2e-8 to 2e-7, as with fp32 FMAs (pieces of 17 bits: 2.5e-7 to 6e-7); its cost, us of 200 int8 sequences as above with 1 / 2 /
// 4 / 8 heads a key: 100 / 99 / 100 / 71 -> 97 / 97 / 102 / 77, none in bf16.
//
// int8 pages: scores are exact integer products (mma .s8) with the query as two int8 terms per element,
// q ~ qs (hi + lo / 128), 14 bits relative to the head's largest component.  Values become fp16 exactly (a byte under
// 0x64 is 1024 + u; as bf16 they take two operations more: 118 us), so the pieces are fp16, of the weight times the row's
// scale.  fp16's range suffices because the running reference that exponents are taken against is not the largest score but
// the largest score + log2(scale): 2^14 times a weight is at most 2^14, and cut off at 2^-38 of the largest so far.
//
// Pipeline: 3 stages of 16 keys per warp, cp.async with zero fill past the last key (a zero weight must not meet
// whatever the shared memory held), page-table entries one tile ahead of their copies.  bf16, 128 wide: 24 KB per
// warp, two CTAs per SM, 128 KB in flight per SM where 36 KB cover the latency.
#pragma once
#include <cuda_fp16.h>

#include "../common/ptx.cuh"
#include "../common/tanh.cuh"

namespace bb {
namespace pdec {

struct Ext {
  float cap_log2;   // 0: no cap; else scores are cap_log2 tanh(scale q.k)
  int window;       // 0: every key
};

__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(live ? 4 : 0) : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t x) {
  uint32_t y;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
  return y;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s8(int (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// First piece of a value: its upper half (eight bits) in bf16, rounded in fp16.  head2: of two values, packed.
// In bf16 all pieces of a weight are above 0, so that they make an infinite value's infinity and not its NaN: what is left
// goes up by tiny(w), 2^-29 of the weight.  (fp16 pieces meet bytes.)
__device__ __forceinline__ float upper(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
template <bool F16>
__device__ __forceinline__ uint32_t head2(float a, float b) {
  if constexpr (F16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
  } else {
    return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
  }
}
template <bool F16>
__device__ __forceinline__ float tiny(float w) { return F16 ? 0.f : fmaxf(w * 0x1p-29f, 0x1p-126f); }
// what the first pieces leave of a, b; ta, tb: tiny of the weights
template <bool F16>
__device__ __forceinline__ float2 rest2(float a, float b, float ta, float tb) {
  if constexpr (F16) {
    const float2 h = __half22float2(__floats2half2_rn(a, b));
    return make_float2(a - h.x, b - h.y);
  } else {
    return make_float2(a - upper(a) + ta, b - upper(b) + tb);
  }
}
// o += a * (pieces).  fp16: a tile's products in one sum (one by one they cost 6 us of the above and gain nothing: the query's
// 14 bits dominate).
template <bool F16, int NP>
__device__ __forceinline__ void add_product(float (&o)[4], const uint32_t (&a)[4], const uint32_t (&b)[NP][2]) {
  constexpr int CHAIN = F16 ? NP : 1;
#pragma unroll
  for (int n0 = NP; n0 > 0; n0 -= CHAIN) {
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int n = n0 - 1; n >= n0 - CHAIN; --n) {
      if constexpr (F16) mma_f16(sum, a, b[n][0], b[n][1]);
      else mma_bf16(sum, a, b[n][0], b[n][1]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) o[j] += sum[j];
  }
}

template <int HD, bool I8>
struct Cfg {
  static constexpr int RB = HD * (I8 ? 1 : 2);       // bytes of a stored row
  static constexpr int CPR = RB / 16;                // 16-byte chunks of it
  static constexpr int NST = 3;
  static constexpr int STAGE = 2 * 16 * RB;          // K rows, V rows
  static constexpr int WARP = NST * STAGE;
  static constexpr int PIPE = 4 * WARP;
  static constexpr int SCALES = I8 ? 4 * NST * 32 * 4 : 0;
  static constexpr int MERGE = 4 * 8 * HD * 4;       // [warp][column][HD], over the pipeline
  static constexpr int SMEM = (PIPE > MERGE ? PIPE : MERGE) + SCALES;
  // chunk c of row r lies where eight consecutive rows of one chunk index cover all banks
  static __device__ __forceinline__ int at(int r, int c) {
    return r * RB + ((CPR >= 8 ? c ^ (r & 7) : c ^ ((r >> 1) & 3)) << 4);
  }
};

__device__ __forceinline__ float ld_peer(uint32_t local, uint32_t rank) {
  float v;
  asm volatile(
      "{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f32 %0, [a];\n\t}"
      : "=f"(v)
      : "r"(local), "r"(rank)
      : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();   // .aligned wants whole warps
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// q: [B, ldq] rows; part_o: fp32 [B, hq, splits, HD], part_ml: fp32 [B, hq, splits, 2] (the exponents' reference in the
// log2 domain, sum); out (when not null: one split, no merge pass): [B, ldo] normalised rows.
template <int HD, int G, bool I8, bool EXT>
__global__ void __launch_bounds__(128, I8 ? 4 : 2)
kernel(const __nv_bfloat16* __restrict__ q, int ldq, const uint8_t* __restrict__ kc, const uint8_t* __restrict__ vc,
       const float* __restrict__ ks, const float* __restrict__ vs, const int* __restrict__ block_tables, int max_blocks,
       const int* __restrict__ seqlens, float* __restrict__ part_o, float* __restrict__ part_ml,
       __nv_bfloat16* __restrict__ out, int ldo, int hq, int hk, int bs, int splits, float scale_log2, int gsplit, Ext x) {
  using C = Cfg<HD, I8>;
  constexpr int PPP = 8 / G < 3 ? 8 / G : 3;    // pieces of the weights in a product: column c carries piece c / G of head c % G
  constexpr int NP = (3 + PPP - 1) / PPP;       // products
  constexpr int MT = HD / 16;          // 16-row tiles of O^T
  constexpr int KS = I8 ? HD / 32 : HD / 16;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ float s_m[4][8], s_l[4][8];

  const int b = blockIdx.x, kvh = blockIdx.y / gsplit, sp = blockIdx.z;
  const int head0 = (kvh * gsplit + blockIdx.y % gsplit) * G;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = lane >> 2, c0 = (lane & 3) * 2;      // fragment row (key, dimension), first of two columns
  pdl_next();
  pdl_wait();
  const int S = seqlens[b];
  const int k_low = EXT && x.window > 0 ? max(S - x.window, 0) : 0;
  const int per_split = ((S - k_low + splits - 1) / splits + 31) / 32 * 32;
  const int k_begin = k_low + sp * per_split;
  const int k_end = min(S, k_begin + per_split);
  const int tiles = k_end > k_begin ? (k_end - k_begin + 15) >> 4 : 0;
  const int* bt = block_tables + (size_t)b * max_blocks;
  const uint32_t pipe = smem_u32(smem) + warp * C::WARP;
  float* scales = reinterpret_cast<float*>(smem + (C::PIPE > C::MERGE ? C::PIPE : C::MERGE)) + warp * C::NST * 32;

  // page row of this lane's key (lane & 15) of a tile, -1 past the last key
  const uint32_t inverse = 0xffffffffu / (uint32_t)bs + 1;    // key / bs = key inverse / 2^32 while key bs < 2^32
  const bool quick = bs > 1 && (uint64_t)max_blocks * bs * bs < (1ull << 32);
  auto page_row = [&](int tile) {
    const int key = k_begin + tile * 16 + (lane & 15);
    const int page = quick ? (int)__umulhi((uint32_t)key, inverse) : key / bs;
    return key < k_end ? (bt[page] * hk + kvh) * bs + key - page * bs : -1;
  };
  auto issue = [&](int stage, int my_row) {
    constexpr int RPP = 32 / C::CPR;   // rows per pass of the warp
    const uint32_t base = pipe + stage * C::STAGE;
    const int c = lane % C::CPR;
#pragma unroll
    for (int p = 0; p < 16 / RPP; ++p) {
      const int r = p * RPP + lane / C::CPR;
      const int pr = __shfl_sync(0xffffffffu, my_row, r);
      const size_t off = (size_t)max(pr, 0) * C::RB + c * 16;
      cp16(base + C::at(r, c), kc + off, pr >= 0);
      cp16(base + 16 * C::RB + C::at(r, c), vc + off, pr >= 0);
    }
    if constexpr (I8)
      cp4(smem_u32(scales + stage * 32 + lane), (lane < 16 ? ks : vs) + max(my_row, 0), my_row >= 0);
  };

  // this warp's tiles: warp, warp + 4, ...
  int next = warp < tiles ? page_row(warp) : -1;
#pragma unroll
  for (int i = 0; i < C::NST - 1; ++i) {
    if (warp + 4 * i < tiles) {
      const int r = next;
      if (warp + 4 * (i + 1) < tiles) next = page_row(warp + 4 * (i + 1));
      issue(i, r);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  // query columns (repeated past the heads)
  const __nv_bfloat16* qh = q + (size_t)b * ldq + (size_t)(head0 + row % G) * HD;
  uint32_t qb[I8 ? 2 : 1][KS][2];
  float col_scale[2];
  if constexpr (I8) {
    float amax = 0.f;
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int j = 0; j < 4; ++j) amax = fmaxf(amax, fabsf(__bfloat162float(qh[s * 32 + h * 16 + c0 * 2 + j])));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float inv = amax > 0.f ? 127.f / amax : 0.f;
    const float qs = amax * (1.f / 127.f) * scale_log2 * (1.f / 128.f);
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t hi = 0, lo = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float f = __bfloat162float(qh[s * 32 + h * 16 + c0 * 2 + j]) * inv;
          const int u = __float2int_rn(f), r = __float2int_rn((f - (float)u) * 128.f);   // |u| <= 127, |r| <= 64
          hi |= (uint32_t)(u & 0xff) << (8 * j);
          lo |= (uint32_t)(r & 0xff) << (8 * j);
        }
        qb[0][s][h] = hi;
        qb[1][s][h] = lo;
      }
    // lane 4 c holds column c's scale
    col_scale[0] = __shfl_sync(0xffffffffu, qs, c0 * 4);
    col_scale[1] = __shfl_sync(0xffffffffu, qs, c0 * 4 + 4);
  } else {
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
      for (int h = 0; h < 2; ++h) qb[0][s][h] = *reinterpret_cast<const uint32_t*>(qh + s * 16 + h * 8 + c0);
    col_scale[0] = col_scale[1] = scale_log2;
  }
  // columns of second (third) pieces
  const bool past1[2] = {c0 >= G, c0 + 1 >= G}, past2[2] = {c0 >= 2 * G, c0 + 1 >= 2 * G};

  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float o[MT][4];
#pragma unroll
  for (int t = 0; t < MT; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) o[t][j] = 0.f;

  int stage = 0;
  for (int tile = warp; tile < tiles; tile += 4) {
    asm volatile("cp.async.wait_group %0;" ::"n"(C::NST - 2) : "memory");
    __syncwarp();                                      // every lane's copies have landed; the last stage read is free
    {
      const int ahead = tile + 4 * (C::NST - 1);
      if (ahead < tiles) {
        const int r = next;
        if (ahead + 4 < tiles) next = page_row(ahead + 4);
        issue((stage + C::NST - 1) % C::NST, r);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const uint32_t sk = pipe + stage * C::STAGE, sv = sk + 16 * C::RB;

    // scores: sc[0], sc[1] of key `row`, sc[2], sc[3] of key row + 8
    float sc[4];
    if constexpr (I8) {
      int hi[4] = {0, 0, 0, 0}, lo[4] = {0, 0, 0, 0};
#pragma unroll
      for (int s = 0; s < KS; ++s) {
        uint32_t a[4];
        ldsm4(a, sk + C::at((lane & 7) + (lane & 8), s * 2 + (lane >> 4)));
        mma_s8(hi, a, qb[0][s][0], qb[0][s][1]);
        mma_s8(lo, a, qb[1][s][0], qb[1][s][1]);
      }
      const float k0 = scales[stage * 32 + row], k1 = scales[stage * 32 + row + 8];
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[j] = (float)(hi[j] * 128 + lo[j]) * col_scale[j & 1] * (j < 2 ? k0 : k1);
    } else {
      float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};   // two chains
#pragma unroll
      for (int s = 0; s < KS; s += 2) {
        uint32_t a[4], a2[4];
        ldsm4(a, sk + C::at((lane & 7) + (lane & 8), s * 2 + (lane >> 4)));
        ldsm4(a2, sk + C::at((lane & 7) + (lane & 8), s * 2 + 2 + (lane >> 4)));
        mma_bf16(s0, a, qb[0][s][0], qb[0][s][1]);
        mma_bf16(s1, a2, qb[0][s + 1][0], qb[0][s + 1][1]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        sc[j] = (s0[j] + s1[j]) * col_scale[0];
        if constexpr (EXT) {
          if (x.cap_log2 > 0.f) sc[j] = x.cap_log2 * tanh_fp32(sc[j]);
        }
      }
    }
    const int left = k_end - (k_begin + tile * 16);     // >= 1
    if (row >= left) sc[0] = sc[1] = -INFINITY;
    if (row + 8 >= left) sc[2] = sc[3] = -INFINITY;

    float mt[2], vscale[2];
    if constexpr (I8) {
      float up[2];                                      // log2 of a row's scale (rows of zeros: -100)
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        vscale[t] = scales[stage * 32 + 16 + row + 8 * t];
        up[t] = fmaxf(__log2f(vscale[t]), -100.f);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) mt[j] = fmaxf(__fadd_ru(sc[j], up[0]), __fadd_ru(sc[j + 2], up[1]));   // no weight above 1
    } else {
      mt[0] = fmaxf(sc[0], sc[2]);
      mt[1] = fmaxf(sc[1], sc[3]);
    }
#pragma unroll
    for (int d = 4; d <= 16; d <<= 1) {
      mt[0] = fmaxf(mt[0], __shfl_xor_sync(0xffffffffu, mt[0], d));
      mt[1] = fmaxf(mt[1], __shfl_xor_sync(0xffffffffu, mt[1], d));
    }
    const bool grown = mt[0] > m[0] || mt[1] > m[1];
    if (__any_sync(0xffffffffu, grown)) {
      float alpha[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float mm = fmaxf(m[j], mt[j]);
        alpha[j] = mm == -INFINITY ? 1.f : exp2f(m[j] - mm);   // every score so far -inf: nothing to rescale
        l[j] *= alpha[j];
        m[j] = mm;
      }
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int j = 0; j < 4; ++j) o[t][j] *= alpha[j & 1];
    }
    // the weights' pieces as the column operand: keys 0..7, keys 8..15
    uint32_t bw[NP][2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      float a = exp2f(sc[2 * t] - m[0]), b = exp2f(sc[2 * t + 1] - m[1]);
      l[0] += a;
      l[1] += b;
      if constexpr (I8) {
        a = a * vscale[t] * 16384.f;
        b = b * vscale[t] * 16384.f;
      }
      const float ta = tiny<I8>(a), tb = tiny<I8>(b);
      const float2 r = rest2<I8>(a, b, ta, tb);
      if constexpr (NP == 3) {
        const float2 r2 = rest2<I8>(r.x, r.y, ta, tb);
        bw[0][t] = head2<I8>(a, b);
        bw[1][t] = head2<I8>(r.x, r.y);
        bw[2][t] = head2<I8>(r2.x, r2.y);
      } else if constexpr (NP == 2) {
        const float2 r2 = rest2<I8>(r.x, r.y, ta, tb);
        bw[0][t] = head2<I8>(past1[0] ? r.x : a, past1[1] ? r.y : b);
        bw[1][t] = head2<I8>(past1[0] ? ta : r2.x, past1[1] ? tb : r2.y);
      } else {
        a = past1[0] ? r.x : a;
        b = past1[1] ? r.y : b;
        const float2 r2 = rest2<I8>(a, b, ta, tb);
        bw[0][t] = head2<I8>(past2[0] ? r2.x : a, past2[1] ? r2.y : b);
      }
    }
#pragma unroll
    for (int n = 0; n < NP; ++n)
#pragma unroll
      for (int t = 0; t < 2; ++t) bw[n][t] = transpose8x8(bw[n][t]);
    if constexpr (I8) {
      // rows r and r + 8 of a 16-row tile are dimensions 2 r and 2 r + 1: the transposing load moves byte pairs
#pragma unroll
      for (int t = 0; t < MT; t += 2) {
        uint32_t v[4];
        ldsm4t(v, sv + C::at((lane & 7) + (lane & 8), t + (lane >> 4)));
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          uint32_t a[4];
          const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));   // 1024 + 128
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t raw = v[u * 2 + h] ^ 0x80808080u;
            const uint32_t ev = __byte_perm(raw, 0x64646464u, 0x4240), od = __byte_perm(raw, 0x64646464u, 0x4341);
            const __half2 fe = __hsub2(*reinterpret_cast<const __half2*>(&ev), bias);
            const __half2 fo = __hsub2(*reinterpret_cast<const __half2*>(&od), bias);
            a[h * 2] = *reinterpret_cast<const uint32_t*>(&fe);
            a[h * 2 + 1] = *reinterpret_cast<const uint32_t*>(&fo);
          }
          add_product<I8>(o[t + u], a, bw);
        }
      }
    } else {
#pragma unroll
      for (int t = 0; t < MT; ++t) {
        uint32_t a[4];
        ldsm4t(a, sv + C::at((lane & 7) + ((lane >> 4) << 3), t * 2 + ((lane >> 3) & 1)));
        add_product<I8>(o[t], a, bw);
      }
    }
    stage = stage + 1 == C::NST ? 0 : stage + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int d = 4; d <= 16; d <<= 1) {
    l[0] += __shfl_xor_sync(0xffffffffu, l[0], d);
    l[1] += __shfl_xor_sync(0xffffffffu, l[1], d);
  }
  __syncthreads();                                      // the pipelines are free: merge buffer
  float* s_o = reinterpret_cast<float*>(smem);
  if (row == 0) {
    s_m[warp][c0] = m[0];
    s_m[warp][c0 + 1] = m[1];
    s_l[warp][c0] = l[0];
    s_l[warp][c0 + 1] = l[1];
  }
#pragma unroll
  for (int t = 0; t < MT; ++t)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int d = I8 ? t * 16 + row * 2 + (j >> 1) : t * 16 + row + (j >> 1) * 8;
      s_o[(warp * 8 + c0 + (j & 1)) * HD + d] = I8 ? o[t][j] * (1.f / 16384.f) : o[t][j];
    }
  __syncthreads();
  // one result per (head, dimension) of this split
  const bool merge = out && splits > 1;                 // the splits of a (sequence, key / value head) are a cluster
  constexpr int PER = (G * HD + 127) / 128;
  __shared__ float f_m[8], f_l[8];
  float kept[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + 128 * k, g = i / HD, c = i % HD;
    if (i >= G * HD) break;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) mm = fmaxf(mm, s_m[w][g]);
    float ll = 0.f, oo = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float a = s_m[w][g] == -INFINITY ? 0.f : exp2f(s_m[w][g] - mm);
      ll += s_l[w][g] * a;
      float sum = 0.f;
#pragma unroll
      for (int k = PPP - 1; k >= 0; --k) sum += s_o[(w * 8 + k * G + g) * HD + c];
      oo += sum * a;
    }
    if (merge) {
      kept[k] = oo;
      if (c == 0) {
        f_m[g] = mm;
        f_l[g] = ll;
      }
    } else if (out) {
      out[(size_t)b * ldo + (size_t)(head0 + g) * HD + c] = __float2bfloat16(ll > 0.f ? oo * (1.f / ll) : 0.f);
    } else {
      const size_t idx = ((size_t)b * hq + head0 + g) * splits + sp;
      part_o[idx * HD + c] = oo;
      if (c == 0) {
        part_ml[idx * 2] = mm;
        part_ml[idx * 2 + 1] = ll;
      }
    }
  }
  if (!merge) return;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < PER; ++k)
    if (threadIdx.x + 128 * k < G * HD) s_o[threadIdx.x + 128 * k] = kept[k];
  cluster_barrier();
  const uint32_t am = smem_u32(f_m), al = smem_u32(f_l), ao = smem_u32(s_o);
  for (int i = threadIdx.x + 128 * sp; i < G * HD; i += 128 * splits) {
    const int g = i / HD, c = i % HD;
    float mm = -INFINITY, ll = 0.f, oo = 0.f;
#pragma unroll 4
    for (int s = 0; s < splits; ++s) mm = fmaxf(mm, ld_peer(am + g * 4, s));
#pragma unroll 4
    for (int s = 0; s < splits; ++s) {
      const float ms = ld_peer(am + g * 4, s), a = ms == -INFINITY ? 0.f : exp2f(ms - mm);
      ll += ld_peer(al + g * 4, s) * a;
      oo += ld_peer(ao + i * 4, s) * a;
    }
    out[(size_t)b * ldo + (size_t)(head0 + g) * HD + c] = __float2bfloat16(oo * (ll > 0.f ? 1.f / ll : 0.f));
  }
  cluster_barrier();                                    // a split's results outlive their readers
}

}  // namespace pdec
}  // namespace bb
