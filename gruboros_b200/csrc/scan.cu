// minGRU recurrence, forward and backward, for sm_100a.
//
//   z_t = sigmoid(k_t),  g(u) = u + 0.5 (u >= 0) | sigmoid(u) (u < 0)
//   h_t = (1 - z_t) * h_{t-1} + z_t * g(u_t),     h_{-1} = h0 (or 0)
//
// This is the linear-space form of the log-space Heinsen scan the reference
// evaluates with softplus / cumsum / logcumsumexp (mingru/minGRU.py:16-28,
// 56-69); all terms are convex combinations of positive numbers, so fp32 in
// linear space is at least as accurate as the reference's fp32 log-space path.
//
// Layout: k, u, h are bf16 [B, T, C] with a row stride (k and u are usually the
// two column halves of one GEMM output).  A cluster of S CTAs (S = 1: one CTA)
// owns 64 channels of one batch row and walks T in rounds of S super-steps, one
// per CTA.  Raw tiles arrive through a 3-stage TMA ring.  Inside a super-step the
// four warps each take a slice of consecutive time steps, scan it locally from a
// zero state (keeping per-step (prefix-product, local value) pairs in registers),
// exchange slice aggregates - through shared memory in one CTA, with st.async
// into every CTA's table (counted on a barrier there) in a cluster - and finish
// with one FMA per element.
// Results go to a per-warp staging tile and leave with one bulk tensor store
// per slice (which also clips the ragged ends of T and C); super-steps that lie
// wholly inside T run a variant of the slice loop without any bounds handling.
// A thread owns two adjacent channels and does their fp32 arithmetic with
// packed instructions (ptx.cuh: ffma2 / fmul2 / fadd2).
#include <type_traits>

#include "ptx.cuh"
#include "tmap.h"
#include "scan.h"
#include "launch.h"

namespace grb {

constexpr int SC_CH = 64;
// Sizes of a kernel of NW warps that each take STEPS time steps of a super-step; NIN tensors in, NOUT tensors out,
// input ring of STAGES super-steps.
template <int NW_, int STEPS_, int STAGES_, int NIN, int NOUT>
struct ScanShape {
  static constexpr int NW = NW_, STEPS = STEPS_, STAGES = STAGES_;
  static constexpr int THREADS = 32 * NW;
  static constexpr int TS = NW * STEPS;                 // time steps of a super-step
  static constexpr int TILE = TS * SC_CH * 2;           // bytes of one tensor tile
  static constexpr int STAGE = NIN * TILE;
  static constexpr int OUT_WARP = NOUT * STEPS * SC_CH * 2;   // staging tiles of one warp
  static constexpr int smem(int S) { return 128 + STAGES * STAGE + NW * OUT_WARP + 1024 * (NW + (S > 1 ? S : 0)) + 64; }
};

__device__ __forceinline__ float ex2f(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcpf(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Both bf16 halves of a word clamped from below at -40 with one instruction (bf16(-40) = 0xC220).  The clamp keeps
// (1 + e^-k)(1 + e^-u) finite (<= e^80 < FLT_MAX); large positive inputs need none: their exponentials flush to zero.
__device__ __forceinline__ uint32_t clamp_below_bf16x2(uint32_t w) {
  uint32_t r;
  asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(w), "r"(0xC220C220u));
  return r;
}

// Forward, both channels of a word at once; k and u already clamped.  Returns a = 1 - z and b = z g(u), z = sigmoid(k).
// Two exponentials and one reciprocal per channel serve both sigmoids.
// u + 0.5 lies above sigmoid(u) exactly where u >= 0 (the sigmoid is concave there and its slope at 0 is 1/4; for
// u < 0 it is convex and stays above its tangent 0.5 + u/4 > 0.5 + u), so g = max of the two; and z sigmoid(u) is
// the shared reciprocal r = 1 / ((1 + e^-k)(1 + e^-u)) itself, so b = max(z (u + 0.5), r).
__device__ __forceinline__ void gate_act_fwd2(uint32_t kk, uint32_t uu, float2& a, float2& b) {
  const float2 c = splat2(-1.4426950408889634f);
  const float2 kf = make_float2(bf16_lo(kk), bf16_hi(kk)), uf = make_float2(bf16_lo(uu), bf16_hi(uu));
  const float2 ka = fmul2(kf, c), ua = fmul2(uf, c);
  const float2 ea = make_float2(ex2f(ka.x), ex2f(ka.y));   // e^{-k}
  const float2 eb = make_float2(ex2f(ua.x), ex2f(ua.y));   // e^{-u}
  const float2 p = fadd2(eb, splat2(1.f));                  // 1 + e^{-u}
  const float2 d = ffma2(ea, p, p);                         // (1 + e^{-k})(1 + e^{-u})
  const float2 r = make_float2(rcpf(d.x), rcpf(d.y));
  const float2 z = fmul2(r, p);
  a = fmul2(ea, z);
  const float2 t = fmul2(z, fadd2(uf, splat2(0.5f)));
  b = make_float2(fmaxf(t.x, r.x), fmaxf(t.y, r.y));
}

// Backward, both channels of a word at once: a = 1 - z, z, g(u) and g'(u).
__device__ __forceinline__ void gate_act_bwd2(uint32_t kk, uint32_t uu, float2& a, float2& z, float2& g, float2& gp) {
  const float2 c = splat2(-1.4426950408889634f);
  const float2 kf = make_float2(bf16_lo(kk), bf16_hi(kk)), uf = make_float2(bf16_lo(uu), bf16_hi(uu));
  const float2 ka = fmul2(kf, c), ua = fmul2(uf, c);
  const float2 ea = make_float2(ex2f(ka.x), ex2f(ka.y));
  const float2 eb = make_float2(ex2f(ua.x), ex2f(ua.y));
  const float2 p = fadd2(eb, splat2(1.f)), q = fadd2(ea, splat2(1.f));
  const float2 d = fmul2(p, q);
  const float2 r = make_float2(rcpf(d.x), rcpf(d.y));
  z = fmul2(r, p);
  const float2 s = fmul2(r, q);                            // sigmoid(u)
  a = fmul2(ea, z);
  const float2 lin = fadd2(uf, splat2(0.5f));
  const float2 ds = fmul2(fmul2(s, eb), s);                // sigmoid'(u)
  const bool p0 = uf.x >= 0.f, p1 = uf.y >= 0.f;
  g = make_float2(p0 ? lin.x : s.x, p1 ? lin.y : s.y);
  gp = make_float2(p0 ? 1.f : ds.x, p1 ? 1.f : ds.y);
}

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const void* desc, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(desc)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}

__device__ __forceinline__ void tma_store_3d(const void* desc, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(desc)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// The staging tile a bulk store was issued from may be rewritten / released once the store has read it.
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// 16 bytes into CTA `cta`'s copy of a shared-memory location, counted on that CTA's copy of `bar`.
__device__ __forceinline__ void st_async(uint32_t addr, uint32_t bar, uint32_t cta, float4 v) {
  asm volatile(
      "{\n"
      ".reg .b32 ra, rb;\n"
      "mapa.shared::cluster.u32 ra, %0, %2;\n"
      "mapa.shared::cluster.u32 rb, %1, %2;\n"
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [ra], {%3, %4, %5, %6}, [rb];\n"
      "}\n" ::"r"(addr), "r"(bar), "r"(cta), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
      : "memory");
}

// What both kernels keep beside the input ring: barriers, and aggregates (prefix product and value, two channels per lane)
// for two rounds: of the CTA's warps, and of the cluster's CTAs.
template <int NW>
struct Exchange {
  uint64_t* full;      // [STAGES] input tiles have landed
  uint64_t* got;       // [2] the aggregates of all CTAs have landed
  float4* loc;         // [2][NW][32]
  float4* all;         // [2][S][32]
  int S, rank;

  __device__ __forceinline__ float4* warp_slot(int par, int w) const { return loc + (par * NW + w) * 32; }
  __device__ __forceinline__ float4* cta_slot(int par, int r) const { return all + (par * S + r) * 32; }
  __device__ __forceinline__ void arm(int par) const { mbar_expect_tx(&got[par], S * 512); }

  // a then b, in the direction of the recurrence
  static __device__ __forceinline__ float4 chain(float4 a, float4 b) {
    return make_float4(a.x * b.x, fmaf(b.x, a.y, b.y), a.z * b.z, fmaf(b.z, a.w, b.w));
  }
  static __device__ __forceinline__ void apply(float4 x, float& c0, float& c1) {
    c0 = fmaf(x.x, c0, x.y);
    c1 = fmaf(x.z, c1, x.w);
  }

  // Publish this warp's aggregate, wait for the others', advance the carried state (c0, c1) over the whole round and return
  // in (in0, in1) the state that enters this warp's slice.  REV: time runs backwards.  False (in every thread of the CTA)
  // when an earlier wait ran out in some thread (ok); its own wait clears ok, for the next round.  A table is written again two rounds later, by warps that have then passed the round between, which
  // every reader of this table enters only after its reads.
  template <bool CL, bool REV>
  __device__ __forceinline__ bool trade(int round, int warp, int lane, float4 mine, bool& ok, float& c0, float& c1,
                                        float& in0, float& in1) const {
    const int par = round & 1;
    warp_slot(par, warp)[lane] = mine;
    if (!__syncthreads_and(ok ? 1 : 0)) return false;
    if constexpr (CL) {
      if (warp < S) {                       // NW >= S: warp d sends the CTA's aggregate to CTA d
        float4 tot = warp_slot(par, REV ? NW - 1 : 0)[lane];
#pragma unroll
        for (int w = 1; w < NW; ++w) tot = chain(tot, warp_slot(par, REV ? NW - 1 - w : w)[lane]);
        st_async(smem_u32(cta_slot(par, rank) + lane), smem_u32(&got[par]), warp, tot);
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&got[par], (round >> 1) & 1))) ok = false;
      if (threadIdx.x == 0) arm(par);
      for (int i = 0; i < S; ++i) {
        const int r = REV ? S - 1 - i : i;
        if (r == rank) { in0 = c0; in1 = c1; }
        apply(cta_slot(par, r)[lane], c0, c1);
      }
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const int w = REV ? NW - 1 - i : i;
        if (REV ? w > warp : w < warp) apply(warp_slot(par, w)[lane], in0, in1);
      }
    } else {
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        const int w = REV ? NW - 1 - i : i;
        if (w == warp) { in0 = c0; in1 = c1; }
        apply(warp_slot(par, w)[lane], c0, c1);
      }
    }
    return true;
  }
};

struct ScanFwdArgs {
  int B, T, C;
  const float* h0;       // [B, C] or null
  __nv_bfloat16* h;      // [B, T, ldh]
  int64_t ldh;
  float* h_last;         // [B, C] or null
  int* err;
};

// TMA_OUT: h leaves through the staging tile and a bulk tensor store (needs a tensor map of h: 16-byte aligned base
// and row stride); otherwise every lane stores its own values.
// CL: launched as clusters of S CTAs along T (x = channel group * S + rank).
template <typename Sh, bool TMA_OUT, bool CL>
__global__ void __launch_bounds__(Sh::THREADS)
scan_fwd_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmU,
                const __grid_constant__ CUtensorMap tmH, const ScanFwdArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  constexpr int STEPS = Sh::STEPS;
  uint8_t* out_stage = smem + Sh::STAGES * Sh::STAGE;                          // [NW][STEPS][64] bf16
  Exchange<Sh::NW> ex;
  ex.S = CL ? static_cast<int>(cluster_size()) : 1;
  ex.rank = CL ? static_cast<int>(cluster_rank()) : 0;
  ex.loc = reinterpret_cast<float4*>(out_stage + Sh::NW * Sh::OUT_WARP);
  ex.all = ex.loc + 2 * Sh::NW * 32;
  ex.full = reinterpret_cast<uint64_t*>(ex.all + (CL ? 2 * ex.S * 32 : 0));
  ex.got = ex.full + Sh::STAGES;
  uint64_t* full = ex.full;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y, c0 = (blockIdx.x / ex.S) * SC_CH;
  const int ch = c0 + 2 * lane;
  const int nss = (p.T + Sh::TS - 1) / Sh::TS;
  const int rounds = (nss + ex.S - 1) / ex.S;

  auto issue = [&](int r) {                     // thread 0: this CTA's super-step of round r (all zeros beyond T)
    const int stage = r % Sh::STAGES, t0 = (r * ex.S + ex.rank) * Sh::TS;
    mbar_expect_tx(&full[stage], Sh::STAGE);
    tma_load_3d(smem + stage * Sh::STAGE, &tmK, &full[stage], c0, t0, b);
    tma_load_3d(smem + stage * Sh::STAGE + Sh::TILE, &tmU, &full[stage], c0, t0, b);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < Sh::STAGES; ++s) mbar_init(&full[s], 1);
    mbar_init(&ex.got[0], 1);
    mbar_init(&ex.got[1], 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmU);
    if (TMA_OUT) tma_prefetch_desc(&tmH);
  }
  if constexpr (CL) cluster_sync();             // every CTA's barriers are ready for the others' aggregates
  else __syncthreads();
  pdl_trigger();
  pdl_wait();
  if (threadIdx.x == 0) {
    if (CL) { ex.arm(0); ex.arm(1); }
    for (int r = 0; r < Sh::STAGES && r < rounds; ++r) issue(r);
  }

  float c_0 = 0.f, c_1 = 0.f;   // carried hidden state of this lane's two channels
  if (p.h0) {
    if (ch < p.C) c_0 = p.h0[static_cast<size_t>(b) * p.C + ch];
    if (ch + 1 < p.C) c_1 = p.h0[static_cast<size_t>(b) * p.C + ch + 1];
  }
  uint32_t* my_stage = reinterpret_cast<uint32_t*>(out_stage + warp * Sh::OUT_WARP) + lane;

  int done = 0;
  bool ok = true;
  for (int r = 0; r < rounds; ++r) {
    const int stage = r % Sh::STAGES;
    const uint32_t phase = (r / Sh::STAGES) & 1;
    const int ss = r * ex.S + ex.rank;
    if (!mbar_wait(&full[stage], phase)) ok = false;

    float2 S[STEPS], P[STEPS];
    const int tbase = ss * Sh::TS + warp * STEPS;
    float4 mine;
    {
      const uint32_t* sk = reinterpret_cast<const uint32_t*>(smem + stage * Sh::STAGE) + (warp * STEPS) * (SC_CH / 2) + lane;
      const uint32_t* su = sk + Sh::TILE / 4;
      float2 sc = splat2(0.f), q = splat2(1.f);
      // local scan of the slice from a zero state; `masked` adds the handling of time steps at or beyond T
      auto slice = [&](auto masked) {
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
          const uint32_t kk = clamp_below_bf16x2(sk[i * (SC_CH / 2)]), uu = clamp_below_bf16x2(su[i * (SC_CH / 2)]);
          float2 a, bb;
          gate_act_fwd2(kk, uu, a, bb);
          if (decltype(masked)::value && tbase + i >= p.T) { a = splat2(1.f); bb = splat2(0.f); }
          sc = ffma2(a, sc, bb);
          q = fmul2(q, a);
          S[i] = sc; P[i] = q;
        }
      };
      if ((ss + 1) * Sh::TS <= p.T) slice(std::false_type{});
      else slice(std::true_type{});
      mine = make_float4(q.x, sc.x, q.y, sc.y);
    }
    float in0, in1;                             // state entering this warp's slice
    if (!ex.template trade<CL, false>(r, warp, lane, mine, ok, c_0, c_1, in0, in1)) break;
    done = r + 1;
    if (threadIdx.x == 0 && r + Sh::STAGES < rounds) issue(r + Sh::STAGES);   // every warp of the CTA has read the stage
    if constexpr (TMA_OUT) {
      if (tbase < p.T) {                        // uniform across the warp
        if (lane == 0) tma_store_wait_read();   // the store issued a super-step ago has read the tile
        __syncwarp();
#pragma unroll
        for (int i = 0; i < STEPS; ++i)
        {
          const float2 v = ffma2(P[i], make_float2(in0, in1), S[i]);
          my_stage[i * (SC_CH / 2)] = pack_bf16(v.x, v.y);
        }
        fence_proxy_async_smem();
        __syncwarp();
        // rows at or beyond T and channels at or beyond C are clipped by the store
        if (lane == 0) tma_store_3d(&tmH, out_stage + warp * Sh::OUT_WARP, c0, tbase, b);
      }
    } else if (ch < p.C) {
      __nv_bfloat16* hp = p.h + (static_cast<size_t>(b) * p.T + tbase) * p.ldh + ch;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        if (tbase + i < p.T) {
          const float v0 = fmaf(P[i].x, in0, S[i].x);
          const float v1 = fmaf(P[i].y, in1, S[i].y);
          if (ch + 1 < p.C) *reinterpret_cast<uint32_t*>(hp + i * p.ldh) = pack_bf16(v0, v1);
          else hp[i * p.ldh] = __float2bfloat16(v0);
        }
      }
    }
  }
  if (TMA_OUT && lane == 0) tma_store_wait_read();   // before the shared memory is released
  if (!ok) atomicExch(p.err, 11);
  if (done < rounds && threadIdx.x == 0)             // a wait ran out: what was issued may still be landing
    for (int r = done; r < rounds && r < done + Sh::STAGES; ++r) mbar_wait(&full[r % Sh::STAGES], (r / Sh::STAGES) & 1);
  if constexpr (CL) cluster_sync();                  // nobody's aggregates land in a CTA that has gone
  if (ex.rank == 0 && warp == 0 && p.h_last) {
    if (ch < p.C) p.h_last[static_cast<size_t>(b) * p.C + ch] = c_0;
    if (ch + 1 < p.C) p.h_last[static_cast<size_t>(b) * p.C + ch + 1] = c_1;
  }
}

struct ScanBwdArgs {
  int B, T, C;
  const float* h0;        // [B, C] or null
  const float* dh_last;   // [B, C] or null: gradient flowing into the final hidden state
  __nv_bfloat16* dk;      // [B, T, ldd]
  __nv_bfloat16* du;      // [B, T, ldd]
  int64_t ldd;
  float* dh0;             // [B, C] or null
  const float* rowscale;  // [B * T] or null: factor applied to row (b, t) of dk and du
  int* err;
};

// Reverse scan.  With a_t = 1 - z_t and G_t = dL/dh_t (direct), define
//   mu_t = a_t * (G_t + mu_{t+1})      (gradient reaching h_{t-1} through step t)
//   lambda_t = G_t + mu_{t+1}          (total gradient of h_t)
//   dk_t = lambda_t * (g(u_t) - h_{t-1}) * z_t * a_t,   du_t = lambda_t * z_t * g'(u_t)
// TMA_OUT (tensor maps of dk and du) and CL as in the forward kernel; the rounds run from the end of T, the time order of
// the CTAs inside a round is the same.
template <typename Sh, bool TMA_OUT, bool CL>
__global__ void __launch_bounds__(Sh::THREADS)
scan_bwd_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmU,
                const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmG,
                const __grid_constant__ CUtensorMap tmDK, const __grid_constant__ CUtensorMap tmDU, const ScanBwdArgs p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  constexpr int STEPS = Sh::STEPS;
  uint8_t* out_stage = smem + Sh::STAGES * Sh::STAGE;                          // [NW][dk, du][STEPS][64] bf16
  Exchange<Sh::NW> ex;
  ex.S = CL ? static_cast<int>(cluster_size()) : 1;
  ex.rank = CL ? static_cast<int>(cluster_rank()) : 0;
  ex.loc = reinterpret_cast<float4*>(out_stage + Sh::NW * Sh::OUT_WARP);
  ex.all = ex.loc + 2 * Sh::NW * 32;
  ex.full = reinterpret_cast<uint64_t*>(ex.all + (CL ? 2 * ex.S * 32 : 0));
  ex.got = ex.full + Sh::STAGES;
  uint64_t* full = ex.full;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y, c0 = (blockIdx.x / ex.S) * SC_CH;
  const int ch = c0 + 2 * lane;
  const int nss = (p.T + Sh::TS - 1) / Sh::TS;
  const int rounds = (nss + ex.S - 1) / ex.S;

  auto issue = [&](int r) {
    const int stage = r % Sh::STAGES, t0 = ((rounds - 1 - r) * ex.S + ex.rank) * Sh::TS;
    uint8_t* s = smem + stage * Sh::STAGE;
    mbar_expect_tx(&full[stage], Sh::STAGE);
    tma_load_3d(s, &tmK, &full[stage], c0, t0, b);
    tma_load_3d(s + Sh::TILE, &tmU, &full[stage], c0, t0, b);
    tma_load_3d(s + 2 * Sh::TILE, &tmH, &full[stage], c0, t0 - 1, b);   // h_{t-1}; row -1 reads zeros
    tma_load_3d(s + 3 * Sh::TILE, &tmG, &full[stage], c0, t0, b);
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < Sh::STAGES; ++s) mbar_init(&full[s], 1);
    mbar_init(&ex.got[0], 1);
    mbar_init(&ex.got[1], 1);
    fence_mbar_init();
    tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmH); tma_prefetch_desc(&tmG);
    if (TMA_OUT) { tma_prefetch_desc(&tmDK); tma_prefetch_desc(&tmDU); }
  }
  if constexpr (CL) cluster_sync();             // every CTA's barriers are ready for the others' aggregates
  else __syncthreads();
  pdl_trigger();
  pdl_wait();
  if (threadIdx.x == 0) {
    if (CL) { ex.arm(0); ex.arm(1); }
    for (int r = 0; r < Sh::STAGES && r < rounds; ++r) issue(r);
  }

  float h00 = 0.f, h01 = 0.f;
  if (p.h0) {
    if (ch < p.C) h00 = p.h0[static_cast<size_t>(b) * p.C + ch];
    if (ch + 1 < p.C) h01 = p.h0[static_cast<size_t>(b) * p.C + ch + 1];
  }
  float m_0 = 0.f, m_1 = 0.f;   // mu carried from later time steps
  if (p.dh_last) {
    if (ch < p.C) m_0 = p.dh_last[static_cast<size_t>(b) * p.C + ch];
    if (ch + 1 < p.C) m_1 = p.dh_last[static_cast<size_t>(b) * p.C + ch + 1];
  }
  uint32_t* my_dk = reinterpret_cast<uint32_t*>(out_stage + warp * Sh::OUT_WARP) + lane;
  uint32_t* my_du = my_dk + Sh::OUT_WARP / 8;

  int done = 0;
  bool ok = true;
  for (int r = 0; r < rounds; ++r) {
    const int ss = (rounds - 1 - r) * ex.S + ex.rank;
    const int stage = r % Sh::STAGES;
    const uint32_t phase = (r / Sh::STAGES) & 1;
    const int tbase = ss * Sh::TS + warp * STEPS;
    const bool inside = ss > 0 && (ss + 1) * Sh::TS <= p.T;     // no step of this super-step is 0 or >= T
    // row scales of this warp's steps, requested before the wait on the tiles so that their latency is hidden
    float rsc[STEPS];
#pragma unroll
    for (int i = 0; i < STEPS; ++i)
      rsc[i] = (p.rowscale && (inside || tbase + i < p.T)) ? __ldg(p.rowscale + static_cast<size_t>(b) * p.T + tbase + i) : 1.f;
    if (!mbar_wait(&full[stage], phase)) ok = false;

    // per step: lambda_loc = G + mu_loc(next), rn = prod of a over later steps of the slice, c1, c2
    float2 L[STEPS], Q[STEPS], C1[STEPS], C2[STEPS];
    float4 mine;
    {
      const uint32_t* sk = reinterpret_cast<const uint32_t*>(smem + stage * Sh::STAGE) + (warp * STEPS) * (SC_CH / 2) + lane;
      const uint32_t* su = sk + Sh::TILE / 4;
      const uint32_t* sh = sk + 2 * (Sh::TILE / 4);
      const uint32_t* sg = sk + 3 * (Sh::TILE / 4);
      float2 mu = splat2(0.f), rr = splat2(1.f);
      auto slice = [&](auto masked) {
        constexpr bool MASKED = decltype(masked)::value;
#pragma unroll
        for (int i = STEPS - 1; i >= 0; --i) {
          const uint32_t kk = clamp_below_bf16x2(sk[i * (SC_CH / 2)]), uu = clamp_below_bf16x2(su[i * (SC_CH / 2)]);
          const uint32_t hh = sh[i * (SC_CH / 2)], gg = sg[i * (SC_CH / 2)];
          float2 a, z, g, d;
          gate_act_bwd2(kk, uu, a, z, g, d);
          float2 hp = make_float2(bf16_lo(hh), bf16_hi(hh));
          float2 G = make_float2(bf16_lo(gg), bf16_hi(gg));
          const int t = tbase + i;
          if (MASKED && t == 0) hp = make_float2(h00, h01);
          float2 c1 = fmul2(ffma2(hp, splat2(-1.f), g), fmul2(z, a));
          float2 c2 = fmul2(z, d);
          if (MASKED && t >= p.T) { a = splat2(1.f); G = splat2(0.f); c1 = splat2(0.f); c2 = splat2(0.f); }
          L[i] = fadd2(G, mu);
          Q[i] = rr;
          C1[i] = c1; C2[i] = c2;
          mu = fmul2(a, L[i]);
          rr = fmul2(rr, a);
        }
      };
      if (inside) slice(std::false_type{});
      else slice(std::true_type{});
      mine = make_float4(rr.x, mu.x, rr.y, mu.y);
    }
    float in0, in1;
    if (!ex.template trade<CL, true>(r, warp, lane, mine, ok, m_0, m_1, in0, in1)) break;
    done = r + 1;
    if (threadIdx.x == 0 && r + Sh::STAGES < rounds) issue(r + Sh::STAGES);
    if constexpr (TMA_OUT) {
      if (tbase < p.T) {                        // uniform across the warp
        if (lane == 0) tma_store_wait_read();   // the stores issued a super-step ago have read the tiles
        __syncwarp();
#pragma unroll
        for (int i = 0; i < STEPS; ++i) {
          const float2 l = fmul2(ffma2(Q[i], make_float2(in0, in1), L[i]), splat2(rsc[i]));
          const float2 vk = fmul2(l, C1[i]), vu = fmul2(l, C2[i]);
          my_dk[i * (SC_CH / 2)] = pack_bf16(vk.x, vk.y);
          my_du[i * (SC_CH / 2)] = pack_bf16(vu.x, vu.y);
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {                        // rows at or beyond T and channels at or beyond C are clipped
          tma_store_3d(&tmDK, out_stage + warp * Sh::OUT_WARP, c0, tbase, b);
          tma_store_3d(&tmDU, out_stage + warp * Sh::OUT_WARP + Sh::OUT_WARP / 2, c0, tbase, b);
        }
      }
    } else if (ch < p.C) {
      const size_t row0 = (static_cast<size_t>(b) * p.T + tbase) * p.ldd + ch;
#pragma unroll
      for (int i = 0; i < STEPS; ++i) {
        if (tbase + i < p.T) {
          const float l0 = fmaf(Q[i].x, in0, L[i].x) * rsc[i];
          const float l1 = fmaf(Q[i].y, in1, L[i].y) * rsc[i];
          const size_t o = row0 + static_cast<size_t>(i) * p.ldd;
          if (ch + 1 < p.C) {
            *reinterpret_cast<uint32_t*>(p.dk + o) = pack_bf16(l0 * C1[i].x, l1 * C1[i].y);
            *reinterpret_cast<uint32_t*>(p.du + o) = pack_bf16(l0 * C2[i].x, l1 * C2[i].y);
          } else {
            p.dk[o] = __float2bfloat16(l0 * C1[i].x);
            p.du[o] = __float2bfloat16(l0 * C2[i].x);
          }
        }
      }
    }
  }
  if (TMA_OUT && lane == 0) tma_store_wait_read();   // before the shared memory is released
  if (!ok) atomicExch(p.err, 12);
  if (done < rounds && threadIdx.x == 0)             // a wait ran out: what was issued may still be landing
    for (int r = done; r < rounds && r < done + Sh::STAGES; ++r) mbar_wait(&full[r % Sh::STAGES], (r / Sh::STAGES) & 1);
  if constexpr (CL) cluster_sync();                  // nobody's aggregates land in a CTA that has gone
  if (ex.rank == 0 && warp == 0 && p.dh0) {
    if (ch < p.C) p.dh0[static_cast<size_t>(b) * p.C + ch] = m_0;
    if (ch + 1 < p.C) p.dh0[static_cast<size_t>(b) * p.C + ch + 1] = m_1;
  }
}

template <int NW, int STEPS, int STAGES> using FwdShape = ScanShape<NW, STEPS, STAGES, 2, 1>;   // k, u -> h
template <int NW, int STEPS, int STAGES> using BwdShape = ScanShape<NW, STEPS, STAGES, 4, 2>;   // k, u, h_prev, g -> dk, du
// One CTA per channel group: four warps with long slices, three CTAs per SM.  Clusters serve launches of few channel groups,
// which are bound by the latency of a round (a slice, two barriers, the trip to the other CTAs: about 3 us), so their CTAs
// have eight warps.  B1 x T2047 x C3072 (48 channel groups): forward 42.6 us on one CTA each, 14.7 us on eight; backward 71.7
// and 25.4 us; B3 x T999 x C3072: 22.8 -> 14.9 and 37.7 -> 26.2 us.
using Fwd1 = FwdShape<4, 16, 3>;
using FwdC = FwdShape<8, 16, 2>;        // sequences of several rounds: half as many rounds as with 8 steps
using FwdCShort = FwdShape<8, 8, 2>;    // short ones: more CTAs have a super-step
using Bwd1 = BwdShape<4, 8, 3>;
using BwdC = BwdShape<8, 8, 2>;
// All (C / 64) x B CTAs of the 1B and 3B shapes are meant to be resident at once: three per SM.
static_assert(3 * (Fwd1::smem(1) + 1024) <= 233472 && 3 * (Bwd1::smem(1) + 1024) <= 233472, "three scan CTAs per SM must fit");

// CTAs per cluster: T is split as long as all clusters fit on the machine at once and each CTA has a super-step of its own.
template <typename Sh, typename Kern>
static int pick_split(Kern kern, int groups, int T) {
  static int fit[4] = {-1, -1, -1, -1};      // clusters of 2, 4, 8 CTAs that are resident together
  const int nss = (T + Sh::TS - 1) / Sh::TS;
  int S = 1;
  for (int i = 1; i < 4; ++i) {
    const int n = 1 << i;
    if (n > nss) break;
    if (fit[i] < 0) {
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::smem(8));
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = n; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(n);
      cfg.blockDim = dim3(Sh::THREADS);
      cfg.dynamicSmemBytes = Sh::smem(n);
      cfg.attrs = at;
      cfg.numAttrs = 1;
      int q = 0;
      fit[i] = cudaOccupancyMaxActiveClusters(&q, kern, &cfg) == cudaSuccess ? q : 0;
    }
    if (groups > fit[i]) break;
    S = n;
  }
  return S;
}

template <typename Sh, typename Kern, typename... Args>
static int launch_scan(Kern kern, size_t& granted, int groups, int B, int S, void* st, const Args&... args) {
  const int smem = Sh::smem(S);
  if (static_cast<size_t>(smem) > granted) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -4;
    granted = smem;
  }
  if (S == 1) {
    // Not overlapped with the kernel before: its blocks would take SMs unevenly as that one drains, and these blocks all have
    // the same work.  B5 x T3000 x C2944 forward + backward 200 us so, 245 overlapped; B8 x T8192 x C3072 671 and 723 us.
    kern<<<dim3(groups, B), Sh::THREADS, smem, reinterpret_cast<cudaStream_t>(st)>>>(args...);
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  return launch_pdl(kern, dim3(groups * S, B), Sh::THREADS, smem, reinterpret_cast<cudaStream_t>(st), S, args...);
}

struct ScanIo {                       // inputs of both directions (h and g are the backward's)
  const void *k, *u; int64_t ldku;
  const void* h; int64_t ldh;
  const void* g; int64_t ldg;
};

template <typename Sh, bool CL>
static int run_fwd(const ScanIo& io, const ScanFwdArgs& a, int S, void* st) {
  CUtensorMap tmK, tmU, tmH;
  int rc = make_tmap_btc_bf16(&tmK, io.k, a.C, a.T, a.B, io.ldku, SC_CH, Sh::TS);
  if (rc) return rc;
  rc = make_tmap_btc_bf16(&tmU, io.u, a.C, a.T, a.B, io.ldku, SC_CH, Sh::TS);
  if (rc) return rc;
  // the output leaves through bulk tensor stores when its layout allows a tensor map (16-byte aligned base and rows)
  const bool tma_out = make_tmap_btc_bf16(&tmH, a.h, a.C, a.T, a.B, a.ldh, SC_CH, Sh::STEPS) == 0;
  if (!tma_out) tmH = tmK;
  static size_t granted[2] = {};
  const int groups = (a.C + SC_CH - 1) / SC_CH;
  return tma_out ? launch_scan<Sh>(scan_fwd_kernel<Sh, true, CL>, granted[1], groups, a.B, S, st, tmK, tmU, tmH, a)
                 : launch_scan<Sh>(scan_fwd_kernel<Sh, false, CL>, granted[0], groups, a.B, S, st, tmK, tmU, tmH, a);
}

template <typename Sh, bool CL>
static int run_bwd(const ScanIo& io, const ScanBwdArgs& a, int S, void* st) {
  CUtensorMap tmK, tmU, tmH, tmG, tmDK, tmDU;
  int rc = make_tmap_btc_bf16(&tmK, io.k, a.C, a.T, a.B, io.ldku, SC_CH, Sh::TS);
  if (rc) return rc;
  rc = make_tmap_btc_bf16(&tmU, io.u, a.C, a.T, a.B, io.ldku, SC_CH, Sh::TS);
  if (rc) return rc;
  rc = make_tmap_btc_bf16(&tmH, io.h, a.C, a.T, a.B, io.ldh, SC_CH, Sh::TS);
  if (rc) return rc;
  rc = make_tmap_btc_bf16(&tmG, io.g, a.C, a.T, a.B, io.ldg, SC_CH, Sh::TS);
  if (rc) return rc;
  const bool tma_out = make_tmap_btc_bf16(&tmDK, a.dk, a.C, a.T, a.B, a.ldd, SC_CH, Sh::STEPS) == 0 &&
                       make_tmap_btc_bf16(&tmDU, a.du, a.C, a.T, a.B, a.ldd, SC_CH, Sh::STEPS) == 0;
  if (!tma_out) tmDK = tmDU = tmK;
  static size_t granted[2] = {};
  const int groups = (a.C + SC_CH - 1) / SC_CH;
  return tma_out ? launch_scan<Sh>(scan_bwd_kernel<Sh, true, CL>, granted[1], groups, a.B, S, st, tmK, tmU, tmH, tmG, tmDK, tmDU, a)
                 : launch_scan<Sh>(scan_bwd_kernel<Sh, false, CL>, granted[0], groups, a.B, S, st, tmK, tmU, tmH, tmG, tmDK, tmDU, a);
}

}  // namespace grb

using namespace grb;

extern "C" int grb_scan_fwd(const void* k, const void* u, int64_t ldku, const float* h0, void* h, int64_t ldh,
                            float* h_last, int B, int T, int C, int* err, void* stream) {
  if (B <= 0 || T <= 0 || C <= 0) return 0;
  if (C % 2) return -20;
  const ScanIo io{k, u, ldku};
  const ScanFwdArgs a{B, T, C, h0, reinterpret_cast<__nv_bfloat16*>(h), ldh, h_last, err};
  const int groups = (C + SC_CH - 1) / SC_CH * B;
  const int S = pick_split<FwdC>(scan_fwd_kernel<FwdC, true, true>, groups, T);
  if (S > 1 && T > S * FwdC::TS) return run_fwd<FwdC, true>(io, a, S, stream);
  const int Ss = pick_split<FwdCShort>(scan_fwd_kernel<FwdCShort, true, true>, groups, T);
  return Ss > 1 ? run_fwd<FwdCShort, true>(io, a, Ss, stream) : run_fwd<Fwd1, false>(io, a, 1, stream);
}

extern "C" int grb_scan_bwd(const void* k, const void* u, int64_t ldku, const void* h, int64_t ldh, const void* g,
                            int64_t ldg, const float* h0, const float* dh_last, void* dk, void* du, int64_t ldd,
                            float* dh0, const float* rowscale, int B, int T, int C, int* err, void* stream) {
  if (B <= 0 || T <= 0 || C <= 0) return 0;
  if (C % 2) return -20;
  const ScanIo io{k, u, ldku, h, ldh, g, ldg};
  const ScanBwdArgs a{B, T, C, h0, dh_last, reinterpret_cast<__nv_bfloat16*>(dk), reinterpret_cast<__nv_bfloat16*>(du), ldd, dh0, rowscale, err};
  const int S = pick_split<BwdC>(scan_bwd_kernel<BwdC, true, true>, (C + SC_CH - 1) / SC_CH * B, T);
  return S > 1 ? run_bwd<BwdC, true>(io, a, S, stream) : run_bwd<Bwd1, false>(io, a, 1, stream);
}
