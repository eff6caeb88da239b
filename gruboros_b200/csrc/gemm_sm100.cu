// Single-CTA bf16 GEMM for sm_100a (tcgen05.mma / TMEM / TMA), for problems too small to fill the machine with the
// 256 x 256 tiles of the CTA-pair kernel (gemm_sm100_2cta.cu).
//
//   D[M,N] = A[M,K] * B[N,K]^T  (fp32 accumulate in tensor memory)
//
// One CTA computes one 128 x 128 tile, or - in a cluster of S CTAs - the tile's share of K; two CTAs fit an SM, so one's
// epilogue runs under the other's main loop.  What bounds these problems is how many SMs have work and the fixed
// latencies around a short main loop, hence the small tile, the split of K over a cluster and an epilogue in which every
// CTA of the cluster finishes its part of the rows:
//   warp 0      TMA producer   (cp.async.bulk.tensor, 128B swizzle, 3-stage ring of 64-deep k-blocks)
//   warp 1      MMA issuer     (tcgen05.mma 128 x 128 x 16, accumulator in TMEM)
//   warps 2..9  epilogue: tcgen05.ld -> the fp32 tile in shared memory (over the drained ring) -> [cluster barrier] ->
//               rows rank, rank + S, ... of the tile, each summed over the cluster's tiles through distributed shared
//               memory in rank order -> fused math -> global.  A warp takes whole rows (512-byte accesses), and its
//               row scales and residual rows are fetched while the main loop runs.
//
// Either operand may be "K-major" (reduction dim contiguous in global memory)
// or "MN-major" (the M/N dim contiguous), so that the forward GEMM, dgrad and
// wgrad of a Linear all read the tensors where they already live:
//   forward  y  = x  W^T : A = x  [M,K]  K-major, B = W [N,K] K-major
//   dgrad    dx = dy W   : A = dy [M,N]  K-major, B = W [N,K] MN-major
//   wgrad    dW = dy^T x : A = dy [M,N] MN-major, B = x [M,K] MN-major
// Ragged edges rely on TMA zero-fill for loads and predicates for stores.
//
// Replaces the cuBLAS calls behind nn.Linear in the reference
// (mingru/minGRU.py:45,71; mingru/minLM.py:17-23,75) and their autograd.
#include "ptx.cuh"
#include "gemm_sm100.h"
#include "tmap.h"
#include "launch.h"
#include "gemm_epilogue.cuh"
#include <cmath>
#include <cstdio>

namespace grb {
namespace tile {

constexpr int BM = 128;
constexpr int BK = 64;            // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int CHUNK_BYTES = 64 * BK * 2;     // one 64(MN) x 64(red) MN-major box: 8 KB
constexpr int NUM_EPI_WARPS = 8;
constexpr int EPI_THREADS = 32 * NUM_EPI_WARPS;
constexpr int NUM_THREADS = 64 + EPI_THREADS;
constexpr int MAX_SPLIT = 8;

// The cross-entropy needs the whole row of up to 256 logits in one tile.
template <int EPI> constexpr int tile_n() { return EPI == EPI_CE ? 256 : 128; }
// Input ring.  DEEP (at most one CTA per SM): 128-deep stages, 192 KB in flight, because a lone CTA is bound by the latency of
// its loads (0.33 us per 64-deep k-block with three of them in flight, 0.13 at full tensor rate).  Otherwise 64-deep stages,
// 96 KB, so that two CTAs share an SM.
template <int BN, bool DEEP> struct Ring {
  static constexpr int KSUB = DEEP && BN == 128 ? 2 : 1;               // 64-deep k-blocks per stage
  static constexpr int STAGES = DEEP && BN > 128 ? 4 : 3;
  static constexpr int SUB = (BM + BN) * BK * 2;
  static constexpr int STAGE = KSUB * SUB;
  static constexpr int BYTES = STAGES * STAGE;
  static constexpr int SMEM = BYTES + 1024 /*align*/ + 256 /*barriers*/ + NUM_EPI_WARPS * 128 * 4;
};

static int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  }
  return n;
}

struct Shape {
  int M, N, K, kb_per;   // kb_per: 64-deep k-blocks per CTA of the cluster
  int* err;              // device error word (0 = ok)
};

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes of CTA `cta`'s copy of a shared-memory location.
__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t cta) {
  float4 v;
  asm volatile(
      "{\n"
      ".reg .b32 ra;\n"
      "mapa.shared::cluster.u32 ra, %4, %5;\n"
      "ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [ra];\n"
      "}\n"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(addr), "r"(cta)
      : "memory");
  return v;
}

// Row r, 16-byte chunk j of the fp32 tile in shared memory (conflict-free for a row per lane and for a lane per chunk).
template <int BN>
__device__ __forceinline__ uint32_t tile_addr(uint32_t base, int r, int j) {
  return base + r * (BN * 4) + ((j ^ (r & 7)) << 4);
}

// Columns 4 j .. 4 j + 3 of four rows of the tile, summed over the S CTAs of the cluster in rank order.
template <int BN>
__device__ __forceinline__ void tile_sum4(uint32_t base, const int (&r)[4], int j, int S, float4 (&v)[4]) {
  if (S == 1) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                   : "=f"(v[k].x), "=f"(v[k].y), "=f"(v[k].z), "=f"(v[k].w) : "r"(tile_addr<BN>(base, r[k], j)) : "memory");
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = ld_cluster(tile_addr<BN>(base, r[k], j), 0);
#pragma unroll 2
  for (int c = 1; c < S; ++c) {
    float4 u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) u[k] = ld_cluster(tile_addr<BN>(base, r[k], j), c);
#pragma unroll
    for (int k = 0; k < 4; ++k) { v[k].x += u[k].x; v[k].y += u[k].y; v[k].z += u[k].z; v[k].w += u[k].w; }
  }
}

// 256-way softmax cross-entropy of four rows held by a warp (their shuffle chains overlap): lane has columns 4 lane .. +3
// and 128 + 4 lane .. +3.  loss_rows[row] = logsumexp(v) - v[label];  dlogits = (softmax - onehot) * alpha * rowscale,
// v = rowscale * acc.
__device__ __forceinline__ void ce_rows(const EpiArgs& e, const float4 (&a)[4], const float4 (&b)[4], const float (&rs)[4],
                                        const int (&label)[4], const int (&row)[4], const bool (&in)[4], int n0, int N, int lane) {
  const auto col = [&](int j) { return n0 + (j >> 2) * 128 + 4 * lane + (j & 3); };
  float v[4][8], mx[4], sum[4], picked[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float t[8] = {a[k].x, a[k].y, a[k].z, a[k].w, b[k].x, b[k].y, b[k].z, b[k].w};
    mx[k] = -INFINITY; sum[k] = 0.f; picked[k] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[k][j] = t[j] * rs[k];
      if (col(j) < N) mx[k] = fmaxf(mx[k], v[k][j]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 4; ++k) mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (col(j) < N) {
        sum[k] += __expf(v[k][j] - mx[k]);
        if (col(j) == label[k]) picked[k] = v[k][j];
      }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
      picked[k] += __shfl_xor_sync(0xffffffffu, picked[k], o);
    }
  const bool vec = (e.ldo & 3) == 0 && (reinterpret_cast<uintptr_t>(e.out0) & 7) == 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (!in[k]) continue;
    const float lse = mx[k] + __logf(sum[k]);
    if (lane == 0 && e.out1) reinterpret_cast<float*>(e.out1)[row[k]] = lse - picked[k];
    if (!e.out0) continue;
    const float dscale = e.alpha * rs[k];
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(e.out0) + static_cast<size_t>(row[k]) * e.ldo;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float p[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) p[j] = (__expf(v[k][4 * h + j] - lse) - (col(4 * h + j) == label[k] ? 1.f : 0.f)) * dscale;
      const int c = col(4 * h);
      if (vec && c + 4 <= N) *reinterpret_cast<uint2*>(d + c) = make_uint2(pack_bf16(p[0], p[1]), pack_bf16(p[2], p[3]));
      else
        for (int j = 0; j < 4; ++j)
          if (c + j < N) d[c + j] = __float2bfloat16(p[j]);
    }
  }
}

// ---------------------------------------------------------------- kernel
template <int MAJ_A, int MAJ_B, int EPI, bool DEEP>
__global__ void __launch_bounds__(NUM_THREADS, DEEP || EPI == EPI_CE ? 1 : 2)
gemm_tile_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Shape s,
                 const EpiArgs e) {
  constexpr int BN = tile_n<EPI>();
  using R = Ring<BN, DEEP>;
  constexpr int STAGES = R::STAGES, KSUB = R::KSUB, A_BYTES = BM * BK * 2;
  static_assert(BM * BN * 4 <= R::BYTES, "the fp32 tile overlays the drained ring");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + R::BYTES);   // [STAGES]
  uint64_t* empty = full + STAGES;                                             // [STAGES]
  uint64_t* tfull = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  float* colsums = reinterpret_cast<float*>(smem + R::BYTES + 256);   // [NUM_EPI_WARPS][128]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t S, rank;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(S));
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));

  // tile -> (m, n): groups of GM m-tiles share their n sweep for L2 reuse
  const int ntm = (s.M + BM - 1) / BM, ntn = (s.N + BN - 1) / BN;
  int tm, tn;
  {
    constexpr int GM = 16;
    const int r = blockIdx.x / S;
    const int per_group = GM * ntn, g = r / per_group, first_m = g * GM;
    const int gsz = min(GM, ntm - first_m), in = r - g * per_group;
    tm = first_m + in % gsz;
    tn = in / gsz;
  }
  const int nkb = (s.K + BK - 1) / BK;
  const int kb0 = rank * s.kb_per, kb1 = min(nkb, kb0 + s.kb_per);     // never empty (host)

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
    mbar_init(tfull, 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  bool ok = true;
  pdl_trigger();
  if (warp != 1) pdl_wait();                  // (the MMA warp touches no global memory)

  // what the epilogue warps fetch while the main loop runs
  constexpr bool PRE = (EPI == EPI_RESID_F32 || EPI == EPI_GELU_BWD);
  const int n0 = tn * BN, row0 = tm * BM;
  const int w = warp - 2;
  const int col = n0 + 4 * lane;
  const int n_ok = min(4, s.N - col);
  const bool vec_ok = (e.ldo & 3) == 0;
  const bool have_pre = PRE && vec_ok && n_ok == 4;
  // rows w * S + rank, + 8 S, ... of the tile; the i-th one's row scale is held by lane i
  const auto tile_row = [&](int i) { return static_cast<int>(w * S + rank + NUM_EPI_WARPS * S * i); };
  float my_scale = 1.f;
  int my_label = 0;
  float4 bv = make_float4(0.f, 0.f, 0.f, 0.f), nw = bv;
  uint4 pre[PRE ? 8 : 1];
  const auto load_aux = [&](int i) {
    uint4 u = make_uint4(0u, 0u, 0u, 0u);
    if constexpr (PRE) {
      const int r = tile_row(i), row = row0 + r;
      if (have_pre && r < BM && row < s.M) {
        const size_t off = static_cast<size_t>(row) * e.ldo + col;
        if constexpr (EPI == EPI_RESID_F32) {
          u = *reinterpret_cast<const uint4*>(reinterpret_cast<const float*>(e.aux) + off);
        } else {
          const uint2 t = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(e.aux) + off);
          u.x = t.x; u.y = t.y;
        }
      }
    }
    return u;
  };

  if (warp == 0) {
    // ------------------------------------------------------ TMA producer
    int stage = 0; uint32_t phase = 0;
    int it = 0;
    for (int kb = kb0; kb < kb1; kb += KSUB, ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(&empty[stage], phase ^ 1))) { ok = false; break; }
      if (lane == 0) {
        const int nsub = min(KSUB, kb1 - kb);
        mbar_expect_tx(&full[stage], nsub * R::SUB);
        for (int sub = 0; sub < nsub; ++sub) {
          uint8_t* sa = smem + stage * R::STAGE + sub * R::SUB;
          uint8_t* sb = sa + A_BYTES;
          const int kk = (kb + sub) * BK;
          if constexpr (MAJ_A == MAJOR_K) {
            tma_load_2d(sa, &tmA, &full[stage], kk, row0);
          } else {
#pragma unroll
            for (int j = 0; j < BM / 64; ++j) tma_load_2d(sa + j * CHUNK_BYTES, &tmA, &full[stage], row0 + 64 * j, kk);
          }
          if constexpr (MAJ_B == MAJOR_K) {
            tma_load_2d(sb, &tmB, &full[stage], kk, n0);
          } else {
#pragma unroll
            for (int j = 0; j < BN / 64; ++j) tma_load_2d(sb + j * CHUNK_BYTES, &tmB, &full[stage], n0 + 64 * j, kk);
          }
        }
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (!ok) {
      // what is still landing gets one bounded wait each before this CTA's shared memory goes away
      if (lane == 0) atomicExch(s.err, 1);
      for (int i = max(0, it - STAGES); i < it; ++i) mbar_wait(&full[i % STAGES], (i / STAGES) & 1);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------- MMA issuer
    constexpr uint32_t idesc = umma_idesc_bf16(BM, BN, MAJ_A == MAJOR_MN, MAJ_B == MAJOR_MN);
    int stage = 0; uint32_t phase = 0;
    for (int kb = kb0; kb < kb1; kb += KSUB) {
      if (!__all_sync(0xffffffffu, mbar_wait(&full[stage], phase))) { ok = false; break; }
      tc_fence_after();
      if (lane == 0) {
        const int nsub = min(KSUB, kb1 - kb);
        for (int sub = 0; sub < nsub; ++sub) {
          const uint32_t sa = smem_u32(smem + stage * R::STAGE + sub * R::SUB);
          const uint32_t sb = sa + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            uint64_t ad, bd;
            if constexpr (MAJ_A == MAJOR_K) ad = umma_smem_desc(sa + k * UMMA_K * 2, 16, 1024);
            else ad = umma_smem_desc(sa + k * UMMA_K * 128, CHUNK_BYTES, 1024);
            if constexpr (MAJ_B == MAJOR_K) bd = umma_smem_desc(sb + k * UMMA_K * 2, 16, 1024);
            else bd = umma_smem_desc(sb + k * UMMA_K * 128, CHUNK_BYTES, 1024);
            umma_bf16(tmem_base, ad, bd, idesc, (kb + sub > kb0 || k > 0) ? 1u : 0u);
          }
        }
        if (kb + KSUB < kb1) umma_commit(&empty[stage]);   // frees the smem stage when the MMAs retire
        else umma_commit(tfull);                           // accumulator complete
      }
      __syncwarp();
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    if (!ok && lane == 0) atomicExch(s.err, 2);
  } else {
    // ------------------------------------------- epilogue: everything that does not need the accumulator
    // row i of the warp: lanes i and i + 16 each add every other partial sum (two fixed chains, so bitwise reproducible)
    const int my_r = tile_row(lane & 15), my_row = row0 + my_r;
    const bool my_in = my_r < BM && my_row < s.M;
    if (e.rowss) {
      if (e.rowss_parts <= 0) {
        if (my_in) my_scale = __ldg(e.rowss + my_row);
      } else {
        const float* p = e.rowss + static_cast<size_t>(my_in ? my_row : 0) * e.rowss_parts;
        float v = 0.f;
#pragma unroll 4
        for (int i = lane >> 4; i < e.rowss_parts; i += 2) v += __ldg(p + i);
        v += __shfl_xor_sync(0xffffffffu, v, 16);
        my_scale = rsqrtf(fmaf(v, e.rowss_inv_d, e.rowss_eps));
      }
      if (e.rstd_out && tn == 0 && lane < 16 && my_in) e.rstd_out[my_row] = my_scale;
    }
    if constexpr (EPI == EPI_CE) my_label = my_in ? reinterpret_cast<const uint8_t*>(e.aux)[my_row] : 0;
    if constexpr (EPI != EPI_CE) {
      if (e.bias && n_ok > 0) {
        bv.x = e.bias[col];
        if (n_ok > 1) bv.y = e.bias[col + 1];
        if (n_ok > 2) bv.z = e.bias[col + 2];
        if (n_ok > 3) bv.w = e.bias[col + 3];
      }
      if (EPI == EPI_RESID_F32 && e.out2 && n_ok > 0) {
        nw.x = e.normw[col];
        if (n_ok > 1) nw.y = e.normw[col + 1];
        if (n_ok > 2) nw.z = e.normw[col + 2];
        if (n_ok > 3) nw.w = e.normw[col + 3];
      }
    }
#pragma unroll
    for (int i = 0; i < (PRE ? 8 : 0); ++i) pre[i] = load_aux(i);

    // ------------------------------------------- accumulator -> shared memory (lane = row)
    ok = __all_sync(0xffffffffu, mbar_wait(tfull, 0));
    if (!ok && lane == 0) atomicExch(s.err, 3);
    tc_fence_after();
    if (ok) {
      const int q = warp & 3;                 // TMEM lane quadrant this warp may read
      const int r = q * 32 + lane;
      const uint32_t base = smem_u32(smem);
#pragma unroll 1
      for (int c = (w >> 2) * (BN / 2); c < ((w >> 2) + 1) * (BN / 2); c += 32) {
        uint32_t v[32];
        tmem_ld32(tmem_base + c + (static_cast<uint32_t>(q * 32) << 16), v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile_addr<BN>(base, r, (c >> 2) + j)), "r"(v[4 * j]),
                       "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                       : "memory");
      }
    }
    tc_fence_before();
    if (S == 1) asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
  }
  if (S > 1) cluster_sync_all();              // every CTA's part of the tile is in its shared memory
  if (warp >= 2) {
    // ------------------------------------------- sum over the cluster, fused math, global (warp = row)
    const uint32_t base = smem_u32(smem);
    const bool good = ok && *reinterpret_cast<volatile int*>(s.err) == 0;   // a failed wait of any role: write nothing
    float cs[4] = {0.f, 0.f, 0.f, 0.f};
    const bool tile_ok = grb_ok(e, tm >= 0 && tm < ntm && tn >= 0 && tn < ntn, GRB_CHK_TILE);
#pragma unroll 1
    for (int i8 = 0; i8 < BM / NUM_EPI_WARPS && tile_row(i8) < BM && good && tile_ok; i8 += 8) {
#pragma unroll
      for (int h = 0; h < 8; h += 4) {
        int r[4], row[4];
        bool in[4];
        float rs[4];
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          r[k] = tile_row(i8 + h + k);
          row[k] = row0 + r[k];
          in[k] = r[k] < BM && row[k] < s.M;
          r[k] = min(r[k], BM - 1);
          rs[k] = __shfl_sync(0xffffffffu, my_scale, (i8 + h + k) & 31);
        }
        if (!in[0]) break;                                   // the rows of a warp ascend
        tile_sum4<BN>(base, r, lane, S, v);
        if constexpr (EPI == EPI_CE) {
          float4 v2[4];
          int label[4];
          tile_sum4<BN>(base, r, lane + 32, S, v2);
#pragma unroll
          for (int k = 0; k < 4; ++k) label[k] = __shfl_sync(0xffffffffu, my_label, (i8 + h + k) & 31);
          ce_rows(e, v, v2, rs, label, row, in, n0, s.N, lane);
        } else {
          float ssq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (in[k] && n_ok > 0)
              epilogue_apply4<EPI>(e, v[k], bv, row[k], col, n_ok, vec_ok, have_pre, pre[PRE ? h + k : 0], rs[k], nw, ssq[k], cs);
          if constexpr (EPI == EPI_RESID_F32) {
            if (e.ssq_out) {
#pragma unroll
              for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < 4; ++k) ssq[k] += __shfl_xor_sync(0xffffffffu, ssq[k], o);
#pragma unroll
              for (int k = 0; k < 4; ++k)
                if (lane == k && in[k] && grb_ok(e, n0 < s.N, GRB_CHK_PARTS)) e.ssq_out[static_cast<size_t>(row[k]) * ntn + tn] = ssq[k];
            }
          }
          if constexpr (PRE) {
            if (i8 + 8 < BM / NUM_EPI_WARPS) {
#pragma unroll
              for (int k = 0; k < 4; ++k) pre[h + k] = load_aux(i8 + 8 + h + k);
            }
          }
        }
      }
    }
    if constexpr (EPI == EPI_GELU_BWD) {
      if (e.colsum) {
        // column sums of the CTA's rows: the warps meet in shared memory, one reduction per column leaves the CTA
#pragma unroll
        for (int j = 0; j < 4; ++j) colsums[w * 128 + 4 * lane + j] = cs[j];
        asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");
        const int c = threadIdx.x - 64;
        if (c < 128 && n0 + c < s.N && good) {
          float t = 0.f;
#pragma unroll
          for (int k = 0; k < NUM_EPI_WARPS; ++k) t += colsums[k * 128 + c];
          atomicAdd(e.colsum + n0 + c, t);
        }
      }
    }
  }

  if (S > 1) cluster_sync_all();              // nobody reads this CTA's shared memory any more
  else __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, BN);
  }
}

// ------------------------------------------------------------------ host
template <int MAJ_A, int MAJ_B, int EPI, bool DEEP>
static int launch_ring(const CUtensorMap& tmA, const CUtensorMap& tmB, const Shape& s, const EpiArgs& e, int S, int grid,
                       cudaStream_t st) {
  auto kern = gemm_tile_kernel<MAJ_A, MAJ_B, EPI, DEEP>;
  constexpr int smem = Ring<tile_n<EPI>(), DEEP>::SMEM;
  static bool attr_done = false;
  if (!attr_done) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -4;
    attr_done = true;
  }
  return launch_pdl(kern, dim3(grid), NUM_THREADS, smem, st, S, tmA, tmB, s, e);
}

template <int MAJ_A, int MAJ_B, int EPI>
static int launch(const void* A, int64_t lda, const void* B, int64_t ldb, int M, int N, int K, int split,
                  const EpiArgs& e, int* err, cudaStream_t st) {
  constexpr int BN = tile_n<EPI>();
  CUtensorMap tmA, tmB;
  int rc;
  // K-major:  global [rows, K]  -> inner = K, outer = rows, box 64 x tile-rows
  // MN-major: global [K, rows]  -> inner = rows, outer = K, box 64 x 64
  if (MAJ_A == MAJOR_K) rc = make_tmap_2d_bf16(&tmA, A, K, M, lda, 64, BM, true);
  else rc = make_tmap_2d_bf16(&tmA, A, M, K, lda, 64, BK, true);
  if (rc) return rc;
  if (MAJ_B == MAJOR_K) rc = make_tmap_2d_bf16(&tmB, B, K, N, ldb, 64, BN, true);
  else rc = make_tmap_2d_bf16(&tmB, B, N, K, ldb, 64, BK, true);
  if (rc) return rc;
  const int nkb = (K + BK - 1) / BK;
  int S = split < 1 ? 1 : split > MAX_SPLIT ? MAX_SPLIT : split;
  if (S > nkb) S = nkb;
  const int kb_per = (nkb + S - 1) / S;
  S = (nkb + kb_per - 1) / kb_per;                        // no CTA without a k-block
  const int64_t grid = static_cast<int64_t>((M + BM - 1) / BM) * ((N + BN - 1) / BN) * S;
  if (grid <= 0) return 0;
  Shape s{M, N, K, kb_per, err};
  EpiArgs ec = e;
  ec.chk_err = err;
  return grid <= num_sms() && kb_per > 4 ? launch_ring<MAJ_A, MAJ_B, EPI, true>(tmA, tmB, s, ec, S, static_cast<int>(grid), st)
                     : launch_ring<MAJ_A, MAJ_B, EPI, false>(tmA, tmB, s, ec, S, static_cast<int>(grid), st);
}

}  // namespace tile
}  // namespace grb

using namespace grb;

// Which kernel a problem goes to: 0 for CTA pairs, else the split of the single-CTA kernel (1, 2 or 4: larger clusters do
// not pack on the GPCs).  The rule compares estimated times (us); its constants are fitted to times measured on a B200 over
// M 296 .. 8188, N 256 .. 8192, K 256 .. 8192 and all epilogues, where the choice was within 15 % of the better one.
//   single CTA: set-up and drain 3.3; 64-deep k-blocks of 32 KB at what L2 gives an SM (0.25 each), for all CTAs of an SM; an
//               epilogue per two CTAs of an SM; barriers and distributed shared memory of a cluster 1.0 (2), 2.4 (4)
//   CTA pair:   set-up and drain 5; k-blocks of a 256 x 256 tile at tensor rate (0.3); epilogues hide under the next tile's
//               main loop as far as that is long enough, the last one does not
// `splitk`: what the pair kernel would be given (> 1 parts, < 0 stream-K).
extern "C" int grb_gemm_plan(int epi, int M, int N, int K, int splitk) {
  static const double epi_tile[8] = {1.5, 1.5, 3.0, 3.0, 3.0, 2.0, 13.0, 2.0};   // by EPI_*
  static const double epi_pair[8] = {3.0, 5.0, 8.0, 10.0, 9.0, 3.5, 0.0, 3.5};
  const double sms = tile::num_sms(), pairs = tile::num_sms() / 2;
  const int nkb = (K + 63) / 64;
  const bool ce = epi == EPI_CE;                                // 128 x 256 tiles, one CTA per SM, rows dominate
  const double tiles = static_cast<double>((M + 127) / 128) * ((N + (ce ? 255 : 127)) / (ce ? 256 : 128));
  double best = 1e30;
  int pick = 1;
  for (int S = 1; S <= 4 && S <= nkb; S *= 2) {
    const int kb = (nkb + S - 1) / S;
    const double ctas = tiles * S, per_sm = ceil(ctas / (S == 4 ? 0.87 * sms : sms));
    const double t = 3.3 + (S == 1 ? 0.0 : S == 2 ? 1.0 : 2.4) + per_sm * kb * (ce ? 0.37 : 0.25) +
                     (ce ? epi_tile[epi] / S * per_sm : epi_tile[epi] * ceil(ctas / (2 * sms)));
    if (t < best) { best = t; pick = S; }
  }
  if (ce) return pick;
  const double ptiles = static_cast<double>((M + 255) / 256) * ((N + 255) / 256);
  double tp;
  if (splitk < 0) {
    tp = 5.0 + ceil(ptiles * nkb / pairs) * 0.3 + 2 * epi_pair[epi];
  } else {
    const int sk = splitk > 1 ? splitk : 1;
    const double waves = ceil(ptiles * sk / pairs), main = (nkb + sk - 1) / sk * 0.3;
    tp = 5.0 + main + (waves - 1) * (main > epi_pair[epi] ? main : epi_pair[epi]) + epi_pair[epi];
  }
  return tp < best ? 0 : pick;
}

extern "C" int grb_gemm(int major_a, int major_b, int epi, const void* A, int64_t lda, const void* B, int64_t ldb,
                        int M, int N, int K, int split, const EpiArgs* e, int* err, int max_ctas, void* stream) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (epi == EPI_CE && N > 256) return -11;
  if (K < 1) return -14;
#define GRB_CASE(MA, MB, EP)                                                   \
  if (major_a == MA && major_b == MB && epi == EP)                             \
    return tile::launch<MA, MB, EP>(A, lda, B, ldb, M, N, K, split, *e, err, st);
  GRB_CASE(MAJOR_K, MAJOR_K, EPI_STORE_BF16)
  GRB_CASE(MAJOR_K, MAJOR_K, EPI_STORE_F32)
  GRB_CASE(MAJOR_K, MAJOR_K, EPI_BIAS_GELU)
  GRB_CASE(MAJOR_K, MAJOR_K, EPI_RESID_F32)
  GRB_CASE(MAJOR_K, MAJOR_K, EPI_CE)
  GRB_CASE(MAJOR_K, MAJOR_MN, EPI_STORE_BF16)
  GRB_CASE(MAJOR_K, MAJOR_MN, EPI_STORE_F32)
  GRB_CASE(MAJOR_K, MAJOR_MN, EPI_GELU_BWD)
  GRB_CASE(MAJOR_MN, MAJOR_MN, EPI_STORE_F32)
  GRB_CASE(MAJOR_MN, MAJOR_MN, EPI_RED_F32)
  GRB_CASE(MAJOR_MN, MAJOR_MN, EPI_RED_SCATTER)
#undef GRB_CASE
  return -12;
}
