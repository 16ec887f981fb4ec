// GEMM of few rows (a decode step's sequences): C[M,N] (op)= alpha * A[M,K] * B[N,K]^T (+ bias[N]), M <= 256.
//
// Such a product is bound by reading the weights B once.  The 128 x BN tiles of gemm_tcgen05.cu put the rows on the
// tensor core's 128 lanes, so a decode step has N / BN tiles: 8 to 64 SMs stream a layer's weights through one TMA
// ring each and the rest idle.  Here the operands change places: 128 output channels of B are the lanes, the rows of A
// (padded to 16) are the columns, and K is cut over the CTAs of a cluster, so that a 1024 x 1024 layer still keeps more
// than a hundred rings in flight.  The cluster adds its partial sums (fp32, s32 for int8) through distributed shared
// memory in rank order: no workspace, no atomics, the same sum on every run.
//
// Reference contracts: crates/kernels/wgsl/{matmul_reg3,matmul_i8_dyn}.wgsl (decode rows of the serving stack).
#include "../common/host.hpp"
#include "../common/ptx.cuh"

namespace bb {
namespace rows {

constexpr int BN = 128;            // weight rows of a tile (tensor core lanes)
constexpr int KB = 128;            // bytes of a k-block: one swizzle row
constexpr int W_BYTES = BN * KB;
constexpr int THREADS = 192;       // warp 0 TMA, warp 1 TMEM + MMA, warps 2..5 epilogue
constexpr int BAR_BYTES = 1024;    // barriers, in front of the ring

struct Args {
  void* C;
  const float* bias;
  const float* scale_m;
  const float* scale_n;
  float alpha;
  int M, N, ldc;
  int ff;              // > 0: B holds gate rows [0, ff) and up rows [ff, 2 ff); C [M, ff] = silu(gate) * up, N = ff
  int rows_pad;        // M rounded up to 16
  int rows_part;       // rows whose sums the ring holds at a time
  int nkb, kb_per;     // k-blocks, k-blocks of a slice
  int slices;          // CTAs of a cluster
  int stages, stage_bytes;
  int tmem_cols;
  int out_mode;        // as GemmArgs::out_mode
  int early;           // B is not written by the kernels before this one: its first blocks load before they end
  int* err;
};

__device__ __forceinline__ uint32_t peer_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ uint4 ld_peer_u4(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void cluster_barrier() {
  __syncwarp();   // .aligned wants whole warps: the loops in front of it may end in the middle of one
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float gelu_tanh(float x) {
  const float k0 = 0.7978845608028654f, k1 = 0.044715f;
  return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
}

// Sums of the cluster's slices, in rank order.
template <bool I8>
__device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
  return I8 ? a + b : __float_as_uint(__uint_as_float(a) + __uint_as_float(b));
}

// Outputs (row, channels of B n .. n + 3, of which `have` exist) from their full sums.
template <bool I8>
__device__ __forceinline__ void scaled4(const Args& a, const uint4& sum, int row, int n, int have, float (&x)[4]) {
  const uint32_t u[4] = {sum.x, sum.y, sum.z, sum.w};
  const float sm = I8 && a.scale_m ? a.scale_m[row] : 1.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    x[j] = (I8 ? (float)(int)u[j] : __uint_as_float(u[j])) * a.alpha;
    if (I8) x[j] *= sm;
    if (I8 && a.scale_n && j < have) x[j] *= a.scale_n[n + j];
    if (a.bias && j < have) x[j] += a.bias[n + j];
    if (a.out_mode == 3) x[j] = gelu_tanh(x[j]);
  }
}
__device__ __forceinline__ void store4(const Args& a, const float (&x)[4], int row, int n, int have) {
  const size_t at = (size_t)row * a.ldc + n;
  if (a.out_mode == 1 || a.out_mode == 2) {
    float* c = static_cast<float*>(a.C) + at;
    if (a.out_mode == 2) {
      for (int j = 0; j < have; ++j) atomicAdd(c + j, x[j]);   // other streams may add to C too
    } else if (have == 4 && (reinterpret_cast<uintptr_t>(c) & 15) == 0) {
      *reinterpret_cast<float4*>(c) = make_float4(x[0], x[1], x[2], x[3]);
    } else {
      for (int j = 0; j < have; ++j) c[j] = x[j];
    }
  } else {
    __nv_bfloat16* c = static_cast<__nv_bfloat16*>(a.C) + at;
    if (have == 4 && (reinterpret_cast<uintptr_t>(c) & 7) == 0) {
      *reinterpret_cast<uint2*>(c) = make_uint2(pack_bf16x2(x[0], x[1]), pack_bf16x2(x[2], x[3]));
    } else {
      for (int j = 0; j < have; ++j) c[j] = __float2bfloat16(x[j]);
    }
  }
}

// GLU: a.ff > 0.
template <bool I8, bool GLU>
__global__ void __launch_bounds__(THREADS, 5)   // three CTAs an SM (split), and registers for the next kernel's
kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x, const Args a) {
  constexpr int BK = I8 ? 128 : 64;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem);
  uint64_t* empty = full + 32;
  uint64_t* done = full + 64;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full + 65);
  uint8_t* ring = smem + BAR_BYTES;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int slice = (int)blockIdx.x % a.slices;
  const int n0 = (int)blockIdx.x / a.slices * (GLU ? BN / 2 : BN);   // first output channel of the tile
  const int kb0 = slice * a.kb_per;
  const int nkb = max(0, min(a.kb_per, a.nkb - kb0));

  if (threadIdx.x == 0) {
    for (int i = 0; i < a.stages; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], 1);
    }
    mbar_init(done, 1);
    mbar_fence_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, a.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_next();                  // after the allocation: a dependent that allocates too cannot get in front
  if (warp > 0 || !a.early) pdl_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      auto load_w = [&](int kb, int st) {
        uint8_t* to = ring + st * a.stage_bytes;
        tma_load_2d(to, &tm_w, &full[st], (kb0 + kb) * BK, n0);
        if (GLU) tma_load_2d(to + W_BYTES / 2, &tm_w, &full[st], (kb0 + kb) * BK, a.ff + n0);
      };
      const int ahead = a.early ? min(nkb, a.stages) : 0;
      for (int kb = 0; kb < ahead; ++kb) {
        mbar_expect_tx(&full[kb], a.stage_bytes);
        load_w(kb, kb);
      }
      if (a.early) pdl_wait();
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(&empty[stage], phase ^ 1)) {
          set_error(a.err, ERR_WAIT_PRODUCER);
          // copies still in flight get a bounded chance to land
          const int last = (stage + a.stages - 1) % a.stages;
          (void)mbar_wait(&full[last], stage == 0 ? phase ^ 1 : phase);
          break;
        }
        uint8_t* s = ring + stage * a.stage_bytes;
        if (kb >= ahead) {
          mbar_expect_tx(&full[stage], a.stage_bytes);
          load_w(kb, stage);
        }
        tma_load_2d(s + W_BYTES, &tm_x, &full[stage], (kb0 + kb) * BK, 0);
        if (++stage == a.stages) stage = 0, phase ^= 1;
      }
    }
    __syncwarp();
    if (a.early) pdl_wait();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = I8 ? umma_idesc(2, 1, 1, 0, 0, BN, a.rows_pad) : umma_idesc(1, 1, 1, 0, 0, BN, a.rows_pad);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int kb = 0; kb < nkb; ++kb) {
        if (!mbar_wait(&full[stage], phase)) {
          set_error(a.err, ERR_WAIT_MMA_FULL);
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sw = smem_u32(ring + stage * a.stage_bytes), sx = sw + W_BYTES;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint64_t dx = umma_smem_desc(sx + k * 32, 16, 1024);
          const uint64_t dw = umma_smem_desc(sw + k * 32, 16, 1024);
          if (I8) umma_i8_ss(tmem, dw, dx, idesc, (kb | k) != 0);
          else umma_f16_ss(tmem, dw, dx, idesc, (kb | k) != 0);
        }
        umma_commit(&empty[stage]);
        if (++stage == a.stages) stage = 0, phase ^= 1;
      }
      if (ok) umma_commit(done);
    }
    __syncwarp();
  }
  // rows_part rows at a time: TMEM -> this slice's sums [row][channel] in the drained ring; then the cluster's CTAs finish
  // the rows in turn, four channels a thread (a warp stores 256 bytes of one row)
  const uint32_t part = smem_u32(ring);
  bool ok = true;
  if (warp >= 2) {
    ok = mbar_wait(done, 0);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok && lane == 0) set_error(a.err, ERR_WAIT_EPILOGUE);
    tc_fence_after();
  }
  for (int r0 = 0; r0 < a.M; r0 += a.rows_part) {
    const int rows = min(a.rows_part, a.M - r0);
    if (warp >= 2) {
      const int quarter = warp & 3;
      for (int c = 0; c < rows && ok; c += 16) {
        uint32_t v[16];
        __syncwarp();
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + r0 + c, v);
        tmem_wait_ld();
        uint32_t* to = reinterpret_cast<uint32_t*>(ring) + (size_t)c * BN + quarter * 32 + lane;
#pragma unroll
        for (int j = 0; j < 16; ++j) to[j * BN] = v[j];
      }
      tc_fence_before();
    }
    if (a.slices > 1) cluster_barrier();
    else __syncthreads();
    auto sums = [&](uint32_t at) {   // at: byte offset in the ring
      if (a.slices == 1) return *reinterpret_cast<const uint4*>(ring + at);
      uint4 sum = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
      for (int s0 = 0; s0 < a.slices; s0 += 4) {   // four reads in flight
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (s0 + j < a.slices) v[j] = ld_peer_u4(peer_addr(part + at, s0 + j));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (s0 + j < a.slices)
            sum = make_uint4(add<I8>(sum.x, v[j].x), add<I8>(sum.y, v[j].y), add<I8>(sum.z, v[j].z), add<I8>(sum.w, v[j].w));
      }
      return sum;
    };
    constexpr int per_row = GLU ? BN / 8 : BN / 4;
#pragma unroll 1
    for (int e = slice * THREADS + (int)threadIdx.x; e < rows * per_row; e += a.slices * THREADS) {
      const int r = e / per_row, ch = (e % per_row) * 4, n = n0 + ch, have = min(4, a.N - n);
      if (have <= 0) continue;
      float x[4];
      scaled4<I8>(a, sums((uint32_t)(r * BN + ch) * 4), r0 + r, n, have, x);
      if constexpr (GLU) {
        float up[4];
        scaled4<I8>(a, sums((uint32_t)(r * BN + BN / 2 + ch) * 4), r0 + r, a.ff + n, have, up);
#pragma unroll
        for (int j = 0; j < 4; ++j) {   // of the values that a bf16 [M, 2 ff] in between would hold
          const float g = __bfloat162float(__float2bfloat16(x[j])), u = __bfloat162float(__float2bfloat16(up[j]));
          x[j] = g / (1.f + __expf(-g)) * u;
        }
      }
      store4(a, x, r0 + r, n, have);
    }
    if (a.slices > 1) cluster_barrier();   // sums outlive their readers
    else __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, a.tmem_cols);
  }
}

template <bool I8, bool GLU>
int launch(const CUtensorMap& tm_w, const CUtensorMap& tm_x, const Args& a, int smem, cudaStream_t stream) {
  static PerDeviceOnce once;
  const cudaError_t e = ensure_dyn_smem(once, kernel<I8, GLU>, 227 * 1024);
  if (e != cudaSuccess) return (int)e;
  constexpr int per = GLU ? BN / 2 : BN;
  const int tiles = (a.N + per - 1) / per;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(tiles * a.slices);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = a.slices;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return launched(cudaLaunchKernelEx(&cfg, kernel<I8, GLU>, tm_w, tm_x, a));
}

// Fills in the ring, the slices that are left of `slices`, and the columns of tensor memory; *smem = shared memory of a CTA.
int plan(Args& a, int K, int bk, int slices, int smem_kb, int* smem) {
  a.rows_pad = (a.M + 15) / 16 * 16;
  a.nkb = (K + bk - 1) / bk;
  a.kb_per = (a.nkb + slices - 1) / slices;
  a.slices = (a.nkb + a.kb_per - 1) / a.kb_per;
  a.stage_bytes = W_BYTES + a.rows_pad * KB;
  const int budget = smem_kb * 1024 - 1024 - BAR_BYTES;
  a.stages = budget / a.stage_bytes;
  if (a.stages > a.kb_per) a.stages = a.kb_per;
  if (a.stages > 32) a.stages = 32;
  if (a.stages < 1) return BB_ESIZE;
  int ring = a.stages * a.stage_bytes;
  if (ring < 16 * BN * 4) ring = 16 * BN * 4;
  a.rows_part = ring / (16 * BN * 4) * 16;
  a.tmem_cols = 32;
  while (a.tmem_cols < a.rows_pad) a.tmem_cols *= 2;
  // A CTA takes at least the share of the SM's shared memory (228 KB, 1 KB of it for each CTA) that its columns are of tensor
  // memory: CTAs that share an SM, other launches' among them, then never ask for more than its 512 columns.  One that waited
  // for columns while its cluster waits for it could wait for a cluster that waits for columns here.
  const int share = a.tmem_cols * (228 * 1024 / 512) - 1024;
  *smem = 1024 + BAR_BYTES + ring;
  if (*smem < share) *smem = share;
  return BB_OK;
}

template <bool I8>
int run(const void* A, const void* B, Args a, int K, int lda, int ldb, int slices, int smem_kb, cudaStream_t stream) {
  constexpr int ES = I8 ? 1 : 2, BK = I8 ? 128 : 64;
  const CUtensorMapDataType dt = I8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  int smem;
  int rc = plan(a, K, BK, slices, smem_kb, &smem);
  if (rc) return rc;
  CUtensorMap tm_w, tm_x;
  rc = make_tmap_2d(&tm_w, dt, ES, B, K, a.ff ? 2 * a.ff : a.N, (uint64_t)ldb * ES, BK, a.ff ? BN / 2 : BN);
  if (rc) return rc;
  rc = make_tmap_2d(&tm_x, dt, ES, A, K, a.M, (uint64_t)lda * ES, BK, a.rows_pad);
  if (rc) return rc;
  return a.ff ? launch<I8, true>(tm_w, tm_x, a, smem, stream) : launch<I8, false>(tm_w, tm_x, a, smem, stream);
}

// Whether this kernel is the faster one.  It re-reads the rows once per 128 channels and adds its slices up afterwards; the
// tiles of gemm_tcgen05.cu walk all of K in one CTA, which takes long where K is long and is over at once where it is short.
// The lines lie where measured sizes cross (8 to 255 rows, 384 to 151936 channels, K 64 to 12288): the form taken is 0.2 %
// behind the faster one in the mean, by more than 8 % at 17 of 1400.  us here / there: 8 x 1024 x 1024 4.1 / 8.6, 48 x 1024 x 768
// 5.2 / 7.5, 40 x 12288 x 256 9.0 / 6.3, 64 x 6144 x 2048 10.3 / 13.8, 128 x 6144 x 4096 17.6 / 22.5, 210 x 6144 x 2048 19.4 / 14.4,
// 210 x 4096 x 4096 16.0 / 22.6, 224 x 4096 x 12288 32 / 60; int8 40 x 6144 x 1024 6.4 / 7.3, 128 x 1024 x 512 8.7 / 6.2, 160 x 6144
// x 4096 14.3 / 15.3, 210 x 6144 x 4096 20.2 / 15.2, 255 x 1024 x 1024 13.7 / 7.3, 255 x 24576 x 4096 50 / 37.
// In a step of dependent launches (early) this kernel's launch, prologue and first weights hide behind the kernel before it, and
// the tiles' do not: about 4.5 us, which shift the lines.  us a decode step, lines of a lone product / these: int8 128 sequences
// of width 4096 592 / 573, 96 of 2048 668 / 651; always this kernel / these: int8 200 (padded to 224) of width 1024 893 / 844, 210
// of 2048 906 / 880.
bool better(int M, int tiles, int nkb, bool i8, bool early) {
  if (M >= 256) return false;
  if (M <= 32) return true;
  const bool wide = tiles > 148;                            // more tiles than SMs: several CTAs of this kernel share one
  if (early && M <= 224) {
    if (i8) return M <= 112 || nkb >= (M <= 160 ? 6 : M <= 208 ? 16 : 32);
    if (M <= 64) return M <= 48 || !wide || nkb >= 32;
    if (tiles <= 48 && nkb >= (M <= 208 ? 32 : 64)) return true;
  }
  if (i8) {
    if (M <= 64) return nkb >= 16 || (nkb >= 8 && tiles <= (M <= 48 ? 48 : 24)) || (wide && nkb >= (M <= 48 ? 3 : 6));
    if (M <= 128) return nkb >= 16 && 2 * tiles <= (M <= 96 ? 6 : 3) * nkb;
    if (M <= 160) return nkb >= 32 || (nkb >= 24 && tiles <= 32);
    return nkb >= 24 && tiles <= (M <= 192 ? nkb : 3 * nkb / 4);
  }
  if (M <= 48) return nkb >= 12 || (nkb >= 8 && tiles <= 48) || (wide && nkb >= 6);
  if (M <= 64) return (nkb >= 8 && tiles <= 48) || (nkb >= 12 && !wide) || nkb >= 32;
  if (M <= 160) return (nkb >= 32 && tiles <= 48) || (nkb >= 64 && M <= 128);
  return nkb >= 32 && (tiles <= 32 || 8 * tiles <= 3 * nkb);
}

// Slices of K and shared memory a CTA.  Many tiles: three CTAs an SM (74 KB hold two or three stages), one to four slices
// as they fit.  Few tiles: slices until one to two CTAs an SM run, at least four k-blocks each; clusters of eight pack a
// GPC badly, so they are left to eight tiles or long K.  Beyond 64 rows a stage is up to 48 KB: an SM to itself where that
// fills the chip, else half an SM.  us at (slices, KB): 64 x 4096 x 1024 (4, 74) 7.7, (8, 74) 9.4; 64 x 12288 x 2048
// (4, 74) 15.2, (2, 110) 16.6; 96 x 3072 x 2048 (4, 220) 9.4, (6, 220) 16.3; int8 200 x 4096 x 12288 (4, 220) 20.8,
// (8, 110) 23.3; 200 x 24576 x 4096 (1, 110) 47, (2, 110) 54.
void split(int M, int tiles, int nkb, int sms, int* slices, int* smem_kb) {
  int s, kb = 74;
  if (tiles > sms / 2) {
    if (M > 128) kb = 110;
    s = (M > 128 ? 3 * sms / 2 : 3 * sms) / tiles;
    if (s > 4) s = 4;
  } else if (M > 64) {
    kb = tiles <= 32 ? 220 : 110;
    s = tiles <= 8 ? 8 : (tiles <= 16 ? 6 : 4);
  } else {
    s = (nkb <= 16 ? sms : (nkb <= 64 ? 3 * sms / 2 : 2 * sms)) / tiles;
    if (tiles > 8 && nkb <= 32 && s > 6) s = 6;
  }
  *slices = s < 1 ? 1 : (s > 8 ? 8 : s);
  *smem_kb = kb;
}

}  // namespace rows
}  // namespace bb

using namespace bb;

// i8: int8 operands with scale_m [M] / scale_n [N] (bf16 out), else bf16 with alpha and bias.  slices (<= 8) of K and smem_kb
// of shared memory a CTA; 0 = chosen by size.  early: B is constant (a served
// model's weights) since before the last launch on this stream that was not a launch_next.  BB_ESIZE: not a shape of this kernel.
static int gemm_rows(const void* A, const void* B, void* C, const float* bias, const float* scale_m, const float* scale_n,
                     int M, int N, int K, int lda, int ldb, int ldc, int i8, int out_mode, float alpha, int slices,
                     int smem_kb, int early, int ff, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return BB_EARG;
  if (M > 256) return BB_ESIZE;
  rows::Args a{};
  a.C = C;
  a.bias = bias;
  a.scale_m = scale_m;
  a.scale_n = scale_n;
  a.alpha = alpha;
  a.M = M;
  a.N = N;
  a.ldc = ldc;
  a.out_mode = out_mode;
  a.early = early;
  a.ff = ff;
  a.err = device_error_word();
  if (slices == 0) {
    const int per = ff ? rows::BN / 2 : rows::BN, tiles = (N + per - 1) / per, nkb = (K + (i8 ? 127 : 63)) / (i8 ? 128 : 64);
    if (!rows::better(M, tiles, nkb, i8, early)) return BB_ESIZE;
    rows::split(M, tiles, nkb, sm_count(), &slices, &smem_kb);
  }
  if (slices < 1 || slices > 8 || smem_kb < 32 || smem_kb > 226) return BB_EARG;
  return i8 ? rows::run<true>(A, B, a, K, lda, ldb, slices, smem_kb, (cudaStream_t)stream)
            : rows::run<false>(A, B, a, K, lda, ldb, slices, smem_kb, (cudaStream_t)stream);
}

BB_API int bb_gemm_rows(const void* A, const void* B, void* C, const float* bias, const float* scale_m, const float* scale_n,
                        int M, int N, int K, int lda, int ldb, int ldc, int i8, int out_mode, float alpha, int slices,
                        int smem_kb, int early, void* stream) {
  return gemm_rows(A, B, C, bias, scale_m, scale_n, M, N, K, lda, ldb, ldc, i8, out_mode, alpha, slices, smem_kb, early, 0, stream);
}

// How gemm_rows would launch these sizes on `sms` SMs: out = slices, bytes of shared memory and columns of tensor memory of a
// CTA.  No device is needed.
BB_API int bb_gemm_rows_plan(int M, int N, int K, int i8, int ff, int sms, int slices, int smem_kb, int* out) {
  if (M <= 0 || N <= 0 || K <= 0 || M > 256) return BB_ESIZE;
  rows::Args a{};
  a.M = M;
  const int bk = i8 ? 128 : 64, per = ff ? rows::BN / 2 : rows::BN;
  if (slices == 0) rows::split(M, (N + per - 1) / per, (K + bk - 1) / bk, sms, &slices, &smem_kb);
  if (slices < 1 || slices > 8 || smem_kb < 32 || smem_kb > 226) return BB_EARG;
  const int rc = rows::plan(a, K, bk, slices, smem_kb, &out[1]);
  out[0] = a.slices;
  out[2] = a.tmem_cols;
  return rc;
}

// C[M, ff] bf16 = silu(A G^T) * (A U^T) for B = [G; U] of ff rows each: a tile is 64 gate and the 64 matching up channels,
// so the product [M, 2 ff] is not written and read again.  The values are those of bb_gemm_rows and bb_swiglu_fwd, which
// took 6.7 us for 1 x 3072 x 1024, 15.6 for 64 x 6144 x 2048, 48 for int8 224 x 12288 x 4096; here 5.8, 14.2, 44.
BB_API int bb_gemm_rows_glu(const void* A, const void* B, void* C, const float* bias, const float* scale_m, const float* scale_n,
                            int M, int ff, int K, int lda, int ldb, int ldc, int i8, int early, void* stream) {
  return gemm_rows(A, B, C, bias, scale_m, scale_n, M, ff, K, lda, ldb, ldc, i8, 0, 1.f, 0, 0, early, ff, stream);
}
