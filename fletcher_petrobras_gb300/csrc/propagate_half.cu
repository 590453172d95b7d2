// Reduced-precision wavefield storage: the step of propagate_fp32.cu with p
// and q stored in 16-bit floats and all arithmetic in FP32.
//
// Storage of one field buffer: (p, q) as a half2 per cell, [z][y][pitch],
// with one power-of-two scale per z-plane: stored = value * 2^e[z].  The
// scale of every new plane comes from the largest magnitudes of the current
// field within 4 planes and of the previous field at that plane, so the new
// values stay below 2^14 (2^16 is FP16's limit) and far above its subnormal
// range.  The FP16X single-shot step sets it itself, plane by plane; the others
// have it set by a small launch before the step.
//
// The extended form (EXT) adds one signed byte per value: the rounding error
// of the half in units of 2^-8 of the half's last place, i.e. a 19-bit
// significand for every value (3 bytes per value).
//
// The CTA is warp-specialised as in propagate_fp32.cu: a producer thread
// issues the TMA loads, the decode warps (three or seven helper warps, RegsH)
// turn the (p, q) halo tile of the arriving plane into an FP32 shared-memory tile, once per
// cell, and evaluate D1y in its halo columns, and TY compute warps run the
// FP32 stencil on it.  The updated plane is encoded with its new scale, and
// the CTA's largest magnitude on it is folded (atomicMax) into the per-plane
// maximum that the next step's scales use; a magnitude beyond FP16's range
// there sets bit 2 of the error word.
//
// What bounds it: FP16 the shared-memory pipe (80% busy) and issue (68%),
// with the FP32 stencil's reads plus the decode; FP16X issue (its decode and
// encode).  272^3 updated cells: FP16 229 us a step, FP16X 275, against 337
// and 377 us when all 16 warps decoded each plane between two CTA-wide
// barriers.  The residual bytes take no conversion instruction (decode,
// encode): 12 of 310 us.  Four decoded tiles instead of three: FP16 244 ->
// 232 us.  Not kept: one barrier for tile and halo columns (FP16 239, FP16X
// 315 us: the compute warps start later), and the halo columns on the
// producer's warp (323 and 372 us: they then wait for the slowest warp).
#include <cuda_fp16.h>
#include <limits.h>

#include "device_util.cuh"
#include "fletcher_internal.h"
#include "stencil_common.cuh"

namespace flt {

template <int TY, bool EXT>
struct GeoH {
  static constexpr int TX = kTileX;
  static constexpr int HX = TX + 2 * kRadius;
  static constexpr int HY = TY + 2 * kRadius;
  static constexpr int HXY = HX * HY;
  static constexpr int NT = TX * TY;
  static constexpr int r128(int b) { return (b + 127) / 128 * 128; }
  static constexpr int HI_B = HXY * 4;                   // half2 halo tile
  static constexpr int LO_B = EXT ? HXY * 2 : 0;         // residual bytes of the halo tile
  static constexpr int ARR_B = kArrivalCoef * NT * 4;
  static constexpr int UPD_B = kUpdateCoef * NT * 4;
  static constexpr int PHI_B = NT * 4;                   // previous field (point box)
  static constexpr int PLO_B = EXT ? HX * TY * 2 : 0;    // its residuals, box from x0-4
  static constexpr int OFF_LO = r128(HI_B);
  static constexpr int OFF_ARR = OFF_LO + r128(LO_B);
  static constexpr int OFF_UPD = OFF_ARR + ARR_B;
  static constexpr int OFF_PHI = OFF_UPD + UPD_B;
  static constexpr int OFF_PLO = OFF_PHI + r128(PHI_B);
  static constexpr int STAGE_B = r128(OFF_PLO + PLO_B);
  static constexpr int H32_B = HXY * 8;                  // one decoded FP32 halo tile
  static constexpr int ROW_B = TY * HX * 8;              // one D1y exchange buffer
  // In-plane terms (A, B) of the last 5 planes.
  static constexpr int AB_B = 5 * NT * 16;
  static_assert(TY % 4 == 0, "tile rows must be a multiple of 4");
  static_assert(ARR_B % 128 == 0 && UPD_B % 128 == 0, "stage regions 128-B aligned");
};


// Shared memory of a CTA: S stages (TMA tiles, the in-plane terms A, B of the
// stage's plane when five stages match their five slots, and a control
// block), then the decoded tiles with their exchange rows.
template <int TY, int S, bool EXT>
struct LayoutH {
  using G = GeoH<TY, EXT>;
  static constexpr bool AB_IN = S == 5;
  static constexpr int AB_SLOT = G::NT * 16;
  static constexpr int OFF_SAB = G::STAGE_B;
  static constexpr int OFF_CTL = OFF_SAB + (AB_IN ? AB_SLOT : 0);
  static constexpr int OFF_HDR = OFF_CTL;         // the item that starts in the stage
  static constexpr int OFF_SCALE = OFF_CTL + 16;  // 2^-e of the arriving plane and of the previous field's
                                                  //   plane of the step, 2^e of the new one
  static constexpr int OFF_FULL = OFF_CTL + 32;   // barriers: loads landed,
  static constexpr int OFF_READY = OFF_CTL + 40;  //   FP32 tile written,
  static constexpr int OFF_HALO = OFF_CTL + 48;   //   halo columns written,
  static constexpr int OFF_EMPTY = OFF_CTL + 56;  //   released by every reader
  static constexpr int OFF_PLANE = OFF_CTL + 64;  // the new plane (-1: none) and its shot (producer only)
  static constexpr int OFF_MAX = OFF_CTL + 72;    // the CTA's largest magnitude on the new plane
  static constexpr int SB = OFF_CTL + 128;
  static constexpr int TILE_B = G::H32_B + G::ROW_B;  // decoded tile, exchange rows
  static constexpr int OFF_TILES = S * SB;
  // Decoded tiles: the decode warps run at most that far ahead.
  static constexpr int REST = S * SB + (AB_IN ? 0 : 5 * AB_SLOT) + 128;
  static constexpr int ND = REST + 4 * TILE_B <= 227 * 1024 ? 4 : 3;
  static constexpr int OFF_AB = OFF_TILES + ND * TILE_B;
  static constexpr size_t BYTES = size_t(REST) + ND * TILE_B;
  static_assert(BYTES <= 227 * 1024, "tile shape exceeds the shared memory of a CTA");
  static_assert(OFF_CTL % 128 == 0 && OFF_TILES % 128 == 0 && TILE_B % 128 == 0 && G::H32_B % 16 == 0 &&
                    OFF_AB % 128 == 0,
                "shared-memory alignment");
};

// Warps and register split (setmaxnreg, which works on warpgroups), as in
// propagate_fp32.cu: TY/4 compute warps and kHelpers/4 helper warps per SM
// sub-partition share what the launch gives them.
// FP16X at 16 rows decodes with seven warps (272^3 updated cells: 311 us a
// step with three of 32 registers, 287 with three of 64, which keep more cells
// in flight, 280 with seven of 32; its compute warps then spill 40 bytes); FP16
// with three (230 us; 246 with 64 registers, its compute warps at 104).
template <int TY, bool EXT>
struct RegsH {
  static constexpr int kHelpers = TY == 16 && EXT ? 8 : 4;  // producer warp + decode warps
  static constexpr int kDecode = kHelpers - 1;
  static constexpr int kThreads = kTileX * (TY + kHelpers);
  static constexpr int kCompute = TY == 16 ? (EXT ? 104 : 112) : TY == 12 ? 152 : 216;
  static constexpr int kHelper = TY == 16 ? 32 : TY == 12 ? 56 : 72;
  static constexpr int kLaunch = TY == 16 ? (EXT ? 80 : 96) : TY == 12 ? 128 : 168;
  static_assert(TY / 4 * kCompute + kHelpers / 4 * kHelper <= (TY + kHelpers) / 4 * kLaunch,
                "the split exceeds the launch's registers");
};

// 2^e as a float (|e| <= 126).
__device__ __forceinline__ float exp2i(int e) { return __int_as_float((127 + e) << 23); }

// The power of two at the leading place of the half h (given as a float),
// at least 2^-14 (FP16's subnormals share the last place of 2^-14).  The
// half's last place is 2^-10 of it, a residual unit 2^-18.
__device__ __forceinline__ float lead(float h) {
  return __int_as_float(max(__float_as_int(h) & 0x7f800000, (127 - 14) << 23));
}

// Value of one stored cell pair: (half + r * 2^-18 * lead(half)) * 2^-e.
// The residual byte r becomes r * 2^-18 without a conversion: r + 128 in the
// last byte of a float in [32, 64), whose last place is 2^-18, less
// 32 + 128 * 2^-18 (both exact).
template <bool EXT>
__device__ __forceinline__ f2 decode(unsigned hv, unsigned short rv, float inv) {
  const float2 h = __half22float2(*reinterpret_cast<const __half2 *>(&hv));
  f2 v = mk2(h.x, h.y);
  if constexpr (EXT) {
    const unsigned u = (unsigned)rv ^ 0x8080u;
    const f2 r = mk2(__uint_as_float(__byte_perm(u, 0x42000000u, 0x7650)),
                     __uint_as_float(__byte_perm(u, 0x42000000u, 0x7651)));
    v = fma2(add2(r, splat(-(32.0f + 128.0f / 262144.0f))), mk2(lead(h.x), lead(h.y)), v);
  }
  return mul2(v, splat(inv));
}

// Stored form of a value pair under scale sc = 2^e.  The residual is rounded
// to an integer (to nearest even) by adding 1.5 * 2^23: the last byte of the
// sum is its two's complement.
template <bool EXT>
__device__ __forceinline__ void encode(f2 v, float sc, unsigned &hv, unsigned short &rv) {
  const f2 a = mul2(v, splat(sc));
  const __half2 h = __floats2half2_rn(lo(a), hi(a));
  hv = *reinterpret_cast<const unsigned *>(&h);
  rv = 0;
  if constexpr (EXT) {
    const float2 hf = __half22float2(h);
    // 2^18 / lead, exact; a - hf is exact, and so is the product.
    const f2 inv = mk2(__uint_as_float((272u << 23) - __float_as_uint(lead(hf.x))),
                       __uint_as_float((272u << 23) - __float_as_uint(lead(hf.y))));
    const f2 d = mul2(sub2(a, mk2(hf.x, hf.y)), inv);
    const f2 r = add2(mk2(fminf(fmaxf(lo(d), -127.f), 127.f), fminf(fmaxf(hi(d), -127.f), 127.f)), splat(12582912.0f));
    rv = (unsigned short)__byte_perm(__float_as_uint(lo(r)), __float_as_uint(hi(r)), 0x0040);
  }
}

// A work item: a z range of the tile column at (x0, y0) of a shot
// (a segment of PropParams::seg).
struct HItem {
  int x0, y0, z0, z1, shot;
};

template <bool BATCH>
__device__ __forceinline__ HItem decode_hitem(int4 w) {
  HItem it;
  it.x0 = BATCH ? kRadius + (w.x & 0xffff) * kTileX : w.x;
  it.y0 = w.y;
  it.z0 = w.z;
  it.z1 = w.w;
  it.shot = BATCH ? int((unsigned)w.x >> 16) : 0;
  return it;
}

// The exponent of a plane of the new field from its largest possible
// magnitude: 4 x the current field's largest magnitude within 4 planes (m_cur,
// float bits), plus the previous field's at that plane, plus 4 x the sources
// near the source plane.
__device__ __forceinline__ int plane_exponent(unsigned m_cur, unsigned m_prev, float src_abs) {
  float b = 4.0f * __uint_as_float(m_cur) + __uint_as_float(m_prev);
  b += 4.0f * src_abs;
  if (!(b > 0.0f)) return 0;
  int ex;
  frexpf(b, &ex);  // b < 2^ex
  return min(max(14 - ex, -100), 100);
}

// Fetches a step's tensor maps into the descriptor cache (the residual
// maps exist in the extended form only).
template <bool EXT>
__device__ __forceinline__ void prefetch_maps(const HalfMaps &m) {
  tma_prefetch_desc(&m.cur_hi);
  tma_prefetch_desc(&m.prev_hi);
  if constexpr (EXT) {
    tma_prefetch_desc(&m.cur_lo);
    tma_prefetch_desc(&m.prev_lo);
  }
  tma_prefetch_desc(&m.arr);
  tma_prefetch_desc(&m.upd);
}

// Loads of step k of an item into one stage: the halo tile of plane k, the
// three in-plane coefficients of plane k while k is in the item's range, and
// for the plane k-4 being updated its seven coefficients and previous field.
template <int TY, bool EXT>
__device__ __forceinline__ void issue_half(unsigned char *stage, uint64_t *bar, const HItem &it, int k,
                                           const HalfMaps &M) {
  using G = GeoH<TY, EXT>;
  const bool center = (k >= it.z0) && (k < it.z1);
  const bool upd = (k - kRadius >= it.z0);
  const uint32_t bytes =
      G::HI_B + G::LO_B + (center ? G::ARR_B : 0) + (upd ? G::UPD_B + G::PHI_B + G::PLO_B : 0);
  mbar_arrive_expect_tx(bar, bytes);
  tma_load_3d(stage, &M.cur_hi, bar, it.x0 - kRadius, it.y0 - kRadius, k);
  if constexpr (EXT) tma_load_3d(stage + G::OFF_LO, &M.cur_lo, bar, it.x0 - kRadius, it.y0 - kRadius, k);
  const int ct = (it.x0 - kRadius) / kTileX;  // tile column in the coefficient block
  if (center) tma_load_4d(stage + G::OFF_ARR, &M.arr, bar, 0, ct, it.y0, k);
  if (upd) {
    tma_load_4d(stage + G::OFF_UPD, &M.upd, bar, kArrivalCoef * kTileX, ct, it.y0, k - kRadius);
    tma_load_3d(stage + G::OFF_PHI, &M.prev_hi, bar, it.x0, it.y0, k - kRadius);
    // 2-byte elements: this box starts at x0-4 so that x * 2 B is a multiple of 16.
    if constexpr (EXT) tma_load_3d(stage + G::OFF_PLO, &M.prev_lo, bar, it.x0 - kRadius, it.y0, k - kRadius);
  }
}

// Whether the step sets the new field's plane exponents itself: the FP16X
// single-shot step, on the producer's warp, ahead of the loads.  Instead of a
// launch before each step (k_half_scales): 128^3 + shell 102.1 -> 98.3 us a
// step, 205 x 129 x 173 82.4 -> 78.5, 56^3 + shell 19.4 -> 18.0, 272^3 279.6 ->
// 274.3.  In FP16, whose stages turn over faster, the slower producer costs
// more than the launch (298 x 249 x 215 190 -> 202 us; on a decode warp
// 236), and in batches the shots' pointers spill (6 shots of 158^3 381 -> 639).
__host__ __device__ constexpr bool own_scales(bool ext, bool batch) { return ext && !batch; }

// BATCH: the items belong to the shots of a batch (P.shots, H.hshots,
// H.hmaps: buffers, exponents and tensor maps by shot).  HOOK: the
// fault-injection variant, as in propagate_fp32.cu.
template <int TY, int S, bool ISO, bool EXT, bool BATCH, bool HOOK = false>
__global__ void __launch_bounds__(RegsH<TY, EXT>::kThreads, 1)
    k_propagate_half(const __grid_constant__ HalfMaps M, const __grid_constant__ HalfParams H) {
  using G = GeoH<TY, EXT>;
  using L = LayoutH<TY, S, EXT>;
  constexpr int kDecodeWarps = RegsH<TY, EXT>::kDecode;
  constexpr bool OWN_SCALES = own_scales(EXT, BATCH);
  const PropParams &P = H.p;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *smem = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
  auto bar = [&](unsigned char *st, int off) { return reinterpret_cast<uint64_t *>(st + off); };
  auto scale_of = [&](unsigned char *st) { return reinterpret_cast<float4 *>(st + L::OFF_SCALE); };
  auto max_of = [&](unsigned char *st) { return reinterpret_cast<unsigned *>(st + L::OFF_MAX); };
  auto plane_of = [&](unsigned char *st) { return reinterpret_cast<int2 *>(st + L::OFF_PLANE); };

  const int tid = threadIdx.x;
  const int lx = tid & 31;
  const int wid = uniform(tid >> 5);
  const int first = P.cta_first[blockIdx.x], nitems = P.cta_first[blockIdx.x + 1] - first;
  if (nitems <= 0) return;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      unsigned char *st = smem + s * L::SB;
      mbar_init(bar(st, L::OFF_FULL), 1);
      mbar_init(bar(st, L::OFF_READY), kDecodeWarps);
      mbar_init(bar(st, L::OFF_HALO), kDecodeWarps);
      mbar_init(bar(st, L::OFF_EMPTY), TY + kDecodeWarps);
      *max_of(st) = 0u;
    }
    mbar_fence_init();
  }
  __syncthreads();
  allow_next_launch();
  wait_previous_launch();
  // Every wait is bounded.
  auto wait = [&](uint64_t *b, uint32_t parity) { return mbar_spin(b, parity, HOOK ? P.wait_tries : kSpinTries); };

  if (wid >= TY) {
    setmaxnreg_dec<RegsH<TY, EXT>::kHelper>();
    const int4 *seg = P.seg + first;
    int stage = 0;
    uint32_t phase = 0;
    if (wid == TY) {
      // ---- producer ----
      // (One thread, or with OWN_SCALES its warp: lane 0 issues and stores.)
      if (!OWN_SCALES && lx != 0) return;
      auto maps_of = [&](int shot) -> const HalfMaps * {
        if constexpr (BATCH) return &H.hmaps[shot].m[P.parity];
        else return &M;
      };
      // What the scales of step k of an item need, by lane, loaded a step ahead:
      // lanes 0..8 the current field's maxima within 4 planes of the plane
      // updated, lane 9 the previous field's, lanes 10 and 11 the exponents of
      // the previous field's plane and of the arriving one.
      auto load_scales = [&](const HItem &it, int k) -> unsigned {
        const int zc = k - kRadius;
        if (lx == 11) return (unsigned)H.e_cur[k];
        if (zc < it.z0) return 0u;
        if (lx == 10) return (unsigned)H.e_prev[zc];
        if (lx == 9) return H.m_prev[zc];
        return lx < 9 ? H.m_cur[zc - kRadius + lx] : 0u;
      };
      // The CTA's maximum on the plane whose step held a stage (every warp
      // has released it) goes to the plane's global maximum.
      auto take_max = [&](unsigned char *st) {
        const unsigned v = *max_of(st);
        *max_of(st) = 0u;
        return v;
      };
      auto fold_max = [&](int2 pl, float sc, unsigned v) {
        if (pl.x < 0 || !v) return;
        unsigned *m = BATCH ? H.hshots[pl.y].Mx + (1 - P.parity) * P.shots[pl.y].sz : H.m_new;
        atomicMax(&m[pl.x], v);
        // Beyond FP16's range: the scale bound was exceeded.
        if (!(__fmul_rn(__uint_as_float(v), sc) < 65504.0f)) atomicOr(P.err, 4u);
      };
      int4 w = seg[0], next = nitems > 1 ? seg[1] : w;
      HItem it = decode_hitem<BATCH>(w);
      int k = it.z0 - kRadius, i = 0, issued = 0;
      unsigned sv = 0u;
      if constexpr (OWN_SCALES) sv = load_scales(it, k);
      if (lx == 0) prefetch_maps<EXT>(*maps_of(it.shot));
      bool ok = true;
      while (i < nitems) {
        // The step's scales, then the next step's loads, before the wait: the
        // issue must follow the stage's release at once.
        const HItem cit = it;
        const int4 cw = w;
        const int ck = k, zc = k - kRadius;
        const bool upd = zc >= it.z0;
        int en = 0;
        float4 scl;
        if constexpr (OWN_SCALES) {
          const ShotDesc &sd = P.one;
          const int zs = sd.src_z >= 0 ? sd.src_z : sd.cor_z;
          const int ec = (int)__shfl_sync(0xffffffffu, sv, 11), ep = (int)__shfl_sync(0xffffffffu, sv, 10);
          en = plane_exponent(__reduce_max_sync(0xffffffffu, lx < 9 && sv <= 0x7f800000u ? sv : 0u),
                              __shfl_sync(0xffffffffu, sv, 9),
                              abs(zc - zs) <= kRadius ? fabsf(P.src) + fabsf(P.cor) : 0.0f);
          scl = make_float4(exp2i(-ec), exp2i(-ep), exp2i(en), 0.0f);
        }
        if (++k >= it.z1 + kRadius && ++i < nitems) {
          w = next;
          it = decode_hitem<BATCH>(w);
          k = it.z0 - kRadius;
          if (i + 1 < nitems) {
            next = seg[i + 1];
            // Batched shots keep their tensor maps in global memory: fetch the
            // next item's into the descriptor cache an item ahead.
            if constexpr (BATCH) prefetch_maps<EXT>(*maps_of(decode_hitem<BATCH>(next).shot));
          }
        }
        if constexpr (OWN_SCALES) {
          if (i < nitems) sv = load_scales(it, k);
        }
        unsigned char *st = smem + stage * L::SB;
        // (The first S waits pass at once: the stage was never filled.)
        if (!wait(bar(st, L::OFF_EMPTY), phase ^ 1u)) {
          ok = false;
          break;
        }
        if (lx == 0) {
          const int2 pl = issued >= S ? *plane_of(st) : make_int2(-1, 0);
          const float sc = scale_of(st)->z;
          const unsigned v = take_max(st);
          fence_proxy_async_smem();
          if (ck == cit.z0 - kRadius) *reinterpret_cast<int4 *>(st + L::OFF_HDR) = cw;
          *plane_of(st) = make_int2(upd ? zc : -1, cit.shot);
          if constexpr (OWN_SCALES) *scale_of(st) = scl;
          if (!HOOK || issued != P.stall_step || blockIdx.x != 0)
            issue_half<TY, EXT>(st, bar(st, L::OFF_FULL), cit, ck, *maps_of(cit.shot));
          fold_max(pl, sc, v);
          if (OWN_SCALES && upd) {
            // Every CTA of the plane finds and stores the same.
            H.e_new[zc] = en;
            H.m_clear[zc] = 0u;
          }
        }
        if constexpr (OWN_SCALES) __syncwarp();
        ++issued;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (lx != 0) {
        if (!ok) atomicOr(P.err, 2u);
        return;
      }
      // The maxima of the last steps, in order.
      for (int a = issued < S ? issued : S; a >= 1 && ok; --a) {
        const int s2 = stage >= a ? stage - a : stage + S - a;
        unsigned char *st = smem + s2 * L::SB;
        if (!wait(bar(st, L::OFF_EMPTY), stage >= a ? phase : phase ^ 1u)) ok = false;
        else fold_max(*plane_of(st), scale_of(st)->z, take_max(st));
      }
      if (!ok) {
        // A bounded wait gave up: wait, bounded, for the loads still in
        // flight into this CTA's stages, then leave (every other thread
        // gives up on its own bounded waits).
        atomicOr(P.err, 2u);
        for (int a = 1; a <= S && a <= issued; ++a) {
          const int s2 = stage >= a ? stage - a : stage + S - a;
          (void)mbar_wait(bar(smem + s2 * L::SB, L::OFF_FULL), stage >= a ? phase : phase ^ 1u, kDrainNs);
        }
      }
      return;
    }
    // ---- decode warps ----
    const int hw = wid - TY - 1;
    const int dt = hw * 32 + lx;  // thread among the decode warps
    constexpr int NDT = 32 * kDecodeWarps;
    const int hxc = (lx & 7) < 4 ? (lx & 7) : G::TX + (lx & 7);  // lane -> halo column, row lane / 8 of a group of 4
    auto decode_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(NDT) : "memory"); };
    [[maybe_unused]] int step = 0;
    int ds = 0;
    int i, k;
    for (i = 0; i < nitems; ++i) {
      const HItem it = decode_hitem<BATCH>(seg[i]);
      const ShotDesc &sd = BATCH ? P.shots[it.shot] : P.one;
      const int src_z = sd.src_z;
      const int kend = it.z1 + kRadius;
      const int *e_cur = H.e_cur, *e_prev = H.e_prev, *e_new = H.e_new;
      if constexpr (BATCH) {
        const int *E = H.hshots[it.shot].E;
        e_cur = E + (H.ecur % 3) * sd.sz;
        e_new = E + ((H.ecur + 1) % 3) * sd.sz;
        e_prev = E + ((H.ecur + 2) % 3) * sd.sz;
      }
      // Exponents of this step's planes, loaded a step ahead.
      int ec = OWN_SCALES ? 0 : e_cur[it.z0 - kRadius], ep = 0, en = 0;
      for (k = it.z0 - kRadius; k < kend; ++k) {
        float inv = exp2i(-ec);
        const float4 ps = make_float4(inv, exp2i(-ep), exp2i(en), 0.0f);
        if (!OWN_SCALES && k + 1 < kend) {
          ec = e_cur[k + 1];
          if (k + 1 - kRadius >= it.z0) {
            ep = e_prev[k + 1 - kRadius];
            en = e_new[k + 1 - kRadius];
          }
        }
        // The decoded tile's last readers: the step L::ND back.
        // (With ND = S that is the step whose stage was refilled.)
        const int es = stage >= L::ND ? stage - L::ND : stage + S - L::ND;
        unsigned char *st = smem + stage * L::SB;
        bool ok = (L::ND == S || wait(bar(smem + es * L::SB, L::OFF_EMPTY), stage >= L::ND ? phase : phase ^ 1u)) &&
                  wait(bar(st, L::OFF_FULL), phase);
        if constexpr (HOOK) ok = ok && !(hw == 1 && blockIdx.x == 0 && step++ == P.quit_step);
        if (!__all_sync(0xffffffffu, ok)) goto gave_up;
        f2 *Hs = reinterpret_cast<f2 *>(smem + L::OFF_TILES + ds * L::TILE_B);
        if constexpr (OWN_SCALES) inv = scale_of(st)->x;
        // Decode once per cell, two cells per thread (one 64-bit load of two
        // half2 cells, one 128-bit store of their FP32 pairs).  The source
        // cell then gains the step's source
        // (original/OpenMP/openmp_insertsource.c:7-13).
        const uint2 *hv2 = reinterpret_cast<const uint2 *>(st);
        const unsigned *rv2 = reinterpret_cast<const unsigned *>(st + G::OFF_LO);
        float4 *Hs4 = reinterpret_cast<float4 *>(Hs);
#pragma unroll
        for (int c0 = 0; c0 < G::HXY / 2; c0 += NDT) {
          const int c2 = c0 + dt;
          if (c0 + NDT <= G::HXY / 2 || c2 < G::HXY / 2) {
            const uint2 h = hv2[c2];
            const unsigned r = EXT ? rv2[c2] : 0u;
            const f2 a = decode<EXT>(h.x, (unsigned short)(r & 0xffffu), inv);
            const f2 b = decode<EXT>(h.y, (unsigned short)(r >> 16), inv);
            Hs4[c2] = make_float4(lo(a), hi(a), lo(b), hi(b));
          }
        }
        if (k == src_z) {
          // Halo-tile index of the source cell, if it lies in this tile.
          const int rx = sd.src_x - (it.x0 - kRadius), ry = sd.src_y - (it.y0 - kRadius);
          if (rx >= 0 && rx < G::HX && ry >= 0 && ry < G::HY) {
            const int src_c = ry * G::HX + rx;
            if (dt == (src_c >> 1) % NDT) Hs[src_c] = add2(Hs[src_c], splat(P.src));
          }
        }
        if (!OWN_SCALES && dt == 0) *scale_of(st) = ps;
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, L::OFF_READY));
        if (k >= it.z0 && k < it.z1) {
          // D1y in the halo columns, from rows that the other decode warps
          // wrote too.
          decode_barrier();
          f2 *db = Hs + G::HXY;
          for (int r = hw * 4 + (lx >> 3); r < TY; r += 4 * kDecodeWarps) {
            const f2 *h = Hs + (r + kRadius) * G::HX + hxc;
            f2 d = mul2(splat(cL1), sub2(h[G::HX], h[-G::HX]));
            d = fma2(splat(cL2), sub2(h[2 * G::HX], h[-2 * G::HX]), d);
            d = fma2(splat(cL3), sub2(h[3 * G::HX], h[-3 * G::HX]), d);
            d = fma2(splat(cL4), sub2(h[4 * G::HX], h[-4 * G::HX]), d);
            db[r * G::HX + hxc] = d;
          }
        }
        __syncwarp();
        if (lx == 0) {
          mbar_arrive(bar(st, L::OFF_HALO));
          mbar_arrive(bar(st, L::OFF_EMPTY));
        }
        if (++ds == L::ND) ds = 0;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    return;
  gave_up:
    // Another decode warp's wait may have succeeded: this one meets the others at
    // every barrier still to come before it leaves (propagate_fp32.cu).
    if (lx == 0) atomicOr(P.err, 1u);
    for (; i < nitems; ++i, k = INT_MIN) {
      const HItem it = decode_hitem<BATCH>(seg[i]);
      for (int z = max(k, it.z0); z < it.z1; ++z) decode_barrier();
    }
    return;
  }

  // ---- compute warps ----
  setmaxnreg_inc<RegsH<TY, EXT>::kCompute>();
  const int ly = wid;
  const float sxy = P.inv_dxy, sxz = P.inv_dxz, syz = P.inv_dyz;
  const float sxx = P.inv_dxx, syy = P.inv_dyy, szz = P.inv_dzz;
  const int ci = ly * G::TX + lx;
  const int hc = (ly + kRadius) * G::HX + (lx + kRadius);
  int stage = 0;
  uint32_t phase = 0;
  int ds = 0;   // decoded tile
  int abw = 0;  // shared A/B ring slot of the arriving plane (the plane 4 back is at abw + 1)
  unsigned char *st = smem;
  for (int item = 0; item < nitems; ++item) {
    if (!wait(bar(st, L::OFF_READY), phase)) {
      atomicOr(P.err, 1u);
      return;
    }
    const HItem it = decode_hitem<BATCH>(uniform4(*reinterpret_cast<const int4 *>(st + L::OFF_HDR)));
    const ShotDesc &sd = BATCH ? P.shots[it.shot] : P.one;
    const int depth = it.z1 - it.z0;
    const int gx = it.x0 + lx;
    const int gy = it.y0 + ly;
    const bool valid = (gx >= sd.bord) && (gx < sd.sx - sd.bord) && (gy >= sd.bord) && (gy < sd.sy - sd.bord);
    const long plane = (long)sd.pitch * sd.sy;
    long at = it.z0 * plane + (long)gy * sd.pitch + gx;
    unsigned *const out_hi = BATCH ? H.hshots[it.shot].hi[1 - P.parity] : H.out_hi;
    unsigned short *const out_lo = BATCH ? H.hshots[it.shot].lo[1 - P.parity] : H.out_lo;
    // The cell that lacks the last step's source, if it is this thread's.
    const int cor_k = (gx == sd.cor_x && gy == sd.cor_y) ? sd.cor_z + kRadius - it.z0 : -1000;

    if (P.skip_rows && (gy < sd.bord || gy >= sd.sy - sd.bord)) {
      // A row outside the updated region: nothing to compute, only the
      // stages to release in step.
      for (int k = -kRadius; k < depth + kRadius; ++k) {
        if (!wait(bar(st, L::OFF_READY), phase)) {
          atomicOr(P.err, 1u);
          return;
        }
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, L::OFF_EMPTY));
        if (!L::AB_IN) abw = abw == 4 ? 0 : abw + 1;
        if (++ds == L::ND) ds = 0;
        st = stage == S - 1 ? smem : st + L::SB;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
      continue;
    }

    f2 Pr[9], Dx[9], Dy[9];

    for (int kb = -kRadius; kb < depth + kRadius; kb += 9) {
#pragma unroll
      for (int j = 0; j < 9; ++j) {
        const int k = kb + j;  // plane, counted from the item's first
        if (k >= depth + kRadius) break;
        if (!wait(bar(st, L::OFF_READY), phase)) {
          atomicOr(P.err, 1u);
          return;
        }
        unsigned char *const st_next = stage == S - 1 ? smem : st + L::SB;
        const bool center = (unsigned)k < (unsigned)depth;
        const bool upd = k >= kRadius;
        f2 *const tile = reinterpret_cast<f2 *>(smem + L::OFF_TILES + ds * L::TILE_B);
        const f2 *Hs = tile + hc;
        const f2 c = Hs[0];
        f2 xa[4], xb[4], ya[4], yb[4];
#pragma unroll
        for (int o = 1; o <= 4; ++o) {
          xa[o - 1] = Hs[o];
          xb[o - 1] = Hs[-o];
          ya[o - 1] = Hs[o * G::HX];
          yb[o - 1] = Hs[-o * G::HX];
        }
        const f2 d1x = d1(xa[0], xb[0], xa[1], xb[1], xa[2], xb[2], xa[3], xb[3]);
        const f2 d1y = d1(ya[0], yb[0], ya[1], yb[1], ya[2], yb[2], ya[3], yb[3]);
        Pr[j] = c;
        Dx[j] = d1x;
        Dy[j] = d1y;
        f2 d2x, d2y;
        f2 *dr = tile + (G::HXY + ly * G::HX + lx + kRadius);
        if (center) {
          d2x = scale<ISO>(d2(c, xa[0], xb[0], xa[1], xb[1], xa[2], xb[2], xa[3], xb[3]), sxx);
          d2y = scale<ISO>(d2(c, ya[0], yb[0], ya[1], yb[1], ya[2], yb[2], ya[3], yb[3]), syy);
          dr[0] = d1y;
        }
        __syncwarp();
        if (upd) {
          const int cs = (j + 5) % 9;
#define RP(o) Pr[(cs + (o)) % 9]
#define RX(o) Dx[(cs + (o)) % 9]
#define RY(o) Dy[(cs + (o)) % 9]
          const f2 d2z = scale<ISO>(d2(RP(0), RP(1), RP(8), RP(2), RP(7), RP(3), RP(6), RP(4), RP(5)), szz);
          const f2 dxz = scale<ISO>(d1(RX(1), RX(8), RX(2), RX(7), RX(3), RX(6), RX(4), RX(5)), sxz);
          const f2 dyz = scale<ISO>(d1(RY(1), RY(8), RY(2), RY(7), RY(3), RY(6), RY(4), RY(5)), syz);
#undef RP
#undef RX
#undef RY
          const float *cu = reinterpret_cast<const float *>(st + G::OFF_UPD) + (ly * (kUpdateCoef * G::TX) + lx);
          const float czz = cu[0], cxz = cu[G::TX], cyz = cu[2 * G::TX];
          const float v2px = cu[3 * G::TX], v2pz = cu[4 * G::TX];
          const float v2sz = cu[5 * G::TX], v2pn = cu[6 * G::TX];
          // (With five slots the plane 4 back is the next one round.)
          const float4 ab = reinterpret_cast<const float4 *>(
              L::AB_IN ? st_next + L::OFF_SAB : smem + L::OFF_AB + (abw == 4 ? 0 : abw + 1) * L::AB_SLOT)[ci];
          const f2 Ak = mk2(ab.x, ab.y), Bk = mk2(ab.z, ab.w);
          const f2 h1 = fma2(splat(cyz), dyz, fma2(splat(cxz), dxz, fma2(splat(czz), d2z, Ak)));
          const f2 h2 = sub2(add2(Bk, d2z), h1);
          const float h1p = lo(h1), h1q = hi(h1), h2p = lo(h2), h2q = hi(h2);
          const float t = __fmul_rn(v2pz, h1q);
          const float rhsp = __fmaf_rn(v2sz, __fsub_rn(h1p, h1q), __fmaf_rn(v2px, h2p, t));
          const float rhsq = __fmaf_rn(-v2sz, __fsub_rn(h2p, h2q), __fmaf_rn(v2pn, h2p, t));
          const unsigned phv = reinterpret_cast<const unsigned *>(st + G::OFF_PHI)[ci];
          unsigned short prv = 0;
          if constexpr (EXT) prv = reinterpret_cast<const unsigned short *>(st + G::OFF_PLO)[ly * G::HX + lx + kRadius];
          const float4 sc = *scale_of(st);
          f2 old = decode<EXT>(phv, prv, sc.y);
          if (k == cor_k) old = add2(old, splat(P.cor));
          const f2 curv = Pr[cs];
          const f2 nw = fma2(mk2(rhsp, rhsq), splat(P.dt2), sub2(add2(curv, curv), old));
          unsigned ohv;
          unsigned short orv;
          encode<EXT>(nw, sc.z, ohv, orv);
          if (valid) {
            out_hi[at] = ohv;
            if constexpr (EXT) out_lo[at] = orv;
          }
          at += plane;
          // The warp's largest magnitude: the bits of non-negative floats
          // order like the floats, so one integer warp reduction finds it
          // (a NaN, above every finite value, reaches the range check).
          unsigned mb = 0u;
          if (valid) mb = max(__float_as_uint(fabsf(lo(nw))), __float_as_uint(fabsf(hi(nw))));
          mb = __reduce_max_sync(0xffffffffu, mb);
          if (lx == 0 && mb) atomicMax(max_of(st), mb);
        }
        if (center) {
          if (!wait(bar(st, L::OFF_HALO), phase)) {
            atomicOr(P.err, 2u);
            return;
          }
          const f2 dxy = scale<ISO>(d1(dr[1], dr[-1], dr[2], dr[-2], dr[3], dr[-3], dr[4], dr[-4]), sxy);
          const float *ca = reinterpret_cast<const float *>(st + G::OFF_ARR) + (ly * (kArrivalCoef * G::TX) + lx);
          const float cxx = ca[0], cyy = ca[G::TX], cxy = ca[2 * G::TX];
          const f2 av = fma2(splat(cxy), dxy, fma2(splat(cyy), d2y, mul2(splat(cxx), d2x)));
          const f2 bv = add2(d2x, d2y);
          reinterpret_cast<float4 *>(L::AB_IN ? st + L::OFF_SAB : smem + L::OFF_AB + abw * L::AB_SLOT)[ci] =
              make_float4(lo(av), hi(av), lo(bv), hi(bv));
        }
        // This warp is done with the stage.
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, L::OFF_EMPTY));
        if (!L::AB_IN) abw = abw == 4 ? 0 : abw + 1;
        if (++ds == L::ND) ds = 0;
        st = st_next;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  }
}

// Before a single-shot step that does not set its own scales: the exponent of
// every plane of the new field, whose maxima are cleared.
__global__ void k_half_scales(const unsigned *m_cur, const unsigned *m_prev, unsigned *m_new, int *e_new, int sz,
                              int src_z, float src_abs) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x;
  allow_next_launch();
  wait_previous_launch();
  if (z >= sz) return;
  float b = 0.0f;
  for (int dz = -kRadius; dz <= kRadius; ++dz)
    if (z + dz >= 0 && z + dz < sz) b = fmaxf(b, __uint_as_float(m_cur[z + dz]));
  e_new[z] = plane_exponent(__float_as_uint(b), m_prev[z], abs(z - src_z) <= kRadius ? src_abs : 0.0f);
  m_new[z] = 0u;
}

// Plane z (= blockIdx.x) of float (p, q) volumes -> stored form, the scale
// from the plane's largest magnitude.
template <bool EXT>
__global__ void k_half_encode_plane(const float *__restrict__ p, const float *__restrict__ q, unsigned *hv,
                                    unsigned short *rv, int *e, unsigned *m, int sx, int sy, int pitch) {
  const int z = blockIdx.x;
  const size_t base = (size_t)z * sx * sy;
  __shared__ float red[32];
  float mx = 0.0f;
  for (int i = threadIdx.x; i < sx * sy; i += blockDim.x) {
    const float a = p ? p[base + i] : 0.f, b = q ? q[base + i] : 0.f;
    mx = fmaxf(mx, fmaxf(fabsf(a), fabsf(b)));
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    mx = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (threadIdx.x == 0) red[0] = mx;
  }
  __syncthreads();
  mx = red[0];
  int ez = 0;
  if (mx > 0.0f) {
    int ex;
    frexpf(mx, &ex);
    ez = min(max(14 - ex, -100), 100);
  }
  if (threadIdx.x == 0) {
    e[z] = ez;
    m[z] = __float_as_uint(mx);
  }
  const float sc = exp2i(ez);
  for (int i = threadIdx.x; i < sx * sy; i += blockDim.x) {
    const int x = i % sx, y = i / sx;
    unsigned h;
    unsigned short l;
    encode<EXT>(mk2(p ? p[base + i] : 0.f, q ? q[base + i] : 0.f), sc, h, l);
    const size_t o = ((size_t)z * sy + y) * pitch + x;
    hv[o] = h;
    if (EXT) rv[o] = l;
  }
}

// One component of a stored volume -> float volume (unpitched).
template <bool EXT>
__global__ void k_half_decode(const unsigned *__restrict__ hv, const unsigned short *__restrict__ rv,
                              const int *__restrict__ e, float *__restrict__ out, int comp, int sx, int sy, int sz,
                              int pitch) {
  const size_t n = (size_t)sx * sy * sz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const size_t x = i % sx, yz = i / sx, z = yz / sy;
    const size_t o = yz * pitch + x;
    const f2 v = decode<EXT>(hv[o], EXT ? rv[o] : (unsigned short)0, exp2i(-e[z]));
    out[i] = comp ? hi(v) : lo(v);
  }
}

// ---- host side ---------------------------------------------------------------

#define FLT_HALF_SHAPES(X) X(12, 4) X(12, 5) X(12, 6) X(8, 6) X(16, 4) X(16, 5)

// Dynamic shared-memory limit of a kernel shape, single-shot or batched
// (once; outside any stream capture before a captured launch).
template <int TY, int S, bool EXT, bool BATCH>
static cudaError_t prepare_half_t() {
  static bool ready = false;
  if (!ready) {
    for (auto kern : {k_propagate_half<TY, S, true, EXT, BATCH>, k_propagate_half<TY, S, false, EXT, BATCH>}) {
      const cudaError_t e =
          prepare_step_kernel((const void *)kern, LayoutH<TY, S, EXT>::BYTES, RegsH<TY, EXT>::kLaunch);
      if (e != cudaSuccess) return e;
    }
    ready = true;
  }
  return cudaSuccess;
}

template <int TY, int S, bool EXT, bool BATCH>
static cudaError_t launch_half_t(const HalfLaunch &L, cudaStream_t s) {
  const cudaError_t e = prepare_half_t<TY, S, EXT, BATCH>();
  if (e != cudaSuccess) return e;
  auto kern = L.h.p.iso ? k_propagate_half<TY, S, true, EXT, BATCH> : k_propagate_half<TY, S, false, EXT, BATCH>;
  return launch_step(kern, L.grid, RegsH<TY, EXT>::kThreads, LayoutH<TY, S, EXT>::BYTES, s, L.m, L.h);
}

// The fault-injection variant: the form's default shape, single shot,
// isotropic grid.  (Any pipeline depth of the step's own shape: the plan and
// the maps depend on the rows only.)
template <bool EXT>
static cudaError_t launch_half_hook(const HalfLaunch &L, cudaStream_t s) {
  constexpr int TY = 16, S = EXT ? 5 : 4;
  if (L.batch || L.tile_rows != TY || !L.h.p.iso) return cudaErrorInvalidValue;
  auto kern = k_propagate_half<TY, S, true, EXT, false, true>;
  const cudaError_t e =
      prepare_step_kernel((const void *)kern, LayoutH<TY, S, EXT>::BYTES, RegsH<TY, EXT>::kLaunch);
  if (e != cudaSuccess) return e;
  return launch_step(kern, L.grid, RegsH<TY, EXT>::kThreads, LayoutH<TY, S, EXT>::BYTES, s, L.m, L.h);
}

bool propagate_half_supported(int tile_rows, int stages) {
#define X(a, b) \
  if (tile_rows == a && stages == b) return true;
  FLT_HALF_SHAPES(X)
#undef X
  return false;
}

cudaError_t propagate_half_launch(const HalfLaunch &L, bool ext, cudaStream_t s) {
  if (!L.batch && !own_scales(ext, false)) {
    const ShotDesc &d = L.h.p.one;
    const cudaError_t e =
        launch_step(k_half_scales, (d.sz + 127) / 128, 128, 0, s, L.h.m_cur, L.h.m_prev, L.h.m_new, L.h.e_new, d.sz,
                    d.src_z >= 0 ? d.src_z : d.cor_z, fabsf(L.h.p.src) + fabsf(L.h.p.cor));
    if (e != cudaSuccess) return e;
  }
  // The work description the chosen kernel reads must be present.
  if (!L.h.p.seg || !L.h.p.cta_first ||
      (L.batch ? (!L.h.p.shots || !L.h.hshots || !L.h.hmaps) : (!L.h.out_hi || !L.h.e_cur)))
    return cudaErrorInvalidValue;
  if (fault_injected(L.h.p)) return ext ? launch_half_hook<true>(L, s) : launch_half_hook<false>(L, s);
#define X(a, b)                                                                                             \
  if (L.tile_rows == a && L.stages == b)                                                                    \
    return ext ? (L.batch ? launch_half_t<a, b, true, true>(L, s) : launch_half_t<a, b, true, false>(L, s)) \
               : (L.batch ? launch_half_t<a, b, false, true>(L, s) : launch_half_t<a, b, false, false>(L, s));
  FLT_HALF_SHAPES(X)
#undef X
  return cudaErrorInvalidValue;
}

cudaError_t propagate_half_prepare(int tile_rows, int stages, bool ext, bool batch) {
#define X(a, b)                                                                                  \
  if (tile_rows == a && stages == b)                                                             \
    return ext ? (batch ? prepare_half_t<a, b, true, true>() : prepare_half_t<a, b, true, false>()) \
               : (batch ? prepare_half_t<a, b, false, true>() : prepare_half_t<a, b, false, false>());
  FLT_HALF_SHAPES(X)
#undef X
  return cudaErrorInvalidValue;
}

// Before each persistent step of a batch: the exponent of every plane of
// every running shot's new field (block i: shot order[i]); the previous
// field's maxima, consumed here, are cleared for the new field's.  The current
// field is in buffer c and uses exponent slot ecur.
__global__ void k_half_scales_batch(const HalfShot *__restrict__ hs, const ShotDesc *__restrict__ sd,
                                    const int *__restrict__ order, int c, int ecur, float src_abs) {
  allow_next_launch();
  wait_previous_launch();
  const int shot = order[blockIdx.x];
  const int sz = sd[shot].sz, src_z = sd[shot].src_z;
  const unsigned *m_cur = hs[shot].Mx + c * sz;
  unsigned *m_prev = hs[shot].Mx + (1 - c) * sz;
  int *e_new = hs[shot].E + ((ecur + 1) % 3) * sz;
  for (int z = threadIdx.x; z < sz; z += blockDim.x) {
    float b = 0.0f;
    for (int dz = -kRadius; dz <= kRadius; ++dz)
      if (z + dz >= 0 && z + dz < sz) b = fmaxf(b, __uint_as_float(m_cur[z + dz]));
    e_new[z] = plane_exponent(__float_as_uint(b), m_prev[z], abs(z - src_z) <= kRadius ? src_abs : 0.0f);
    m_prev[z] = 0u;
  }
}

cudaError_t half_scales_batch(const HalfShot *hs, const ShotDesc *sd, const int *order, int active, int c, int ecur,
                              float src_abs, cudaStream_t s) {
  return launch_step(k_half_scales_batch, active, 256, 0, s, hs, sd, order, c, ecur, src_abs);
}

cudaError_t half_encode(const float *p, const float *q, unsigned *hv, unsigned short *rv, int *e, unsigned *m, int sx,
                        int sy, int sz, int pitch, bool ext, cudaStream_t s) {
  if (ext)
    k_half_encode_plane<true><<<sz, 256, 0, s>>>(p, q, hv, rv, e, m, sx, sy, pitch);
  else
    k_half_encode_plane<false><<<sz, 256, 0, s>>>(p, q, hv, rv, e, m, sx, sy, pitch);
  return cudaGetLastError();
}

cudaError_t half_decode(const unsigned *hv, const unsigned short *rv, const int *e, float *out, int comp, int sx,
                        int sy, int sz, int pitch, bool ext, int grid, cudaStream_t s) {
  if (ext)
    k_half_decode<true><<<grid, 256, 0, s>>>(hv, rv, e, out, comp, sx, sy, sz, pitch);
  else
    k_half_decode<false><<<grid, 256, 0, s>>>(hv, rv, e, out, comp, sx, sy, sz, pitch);
  return cudaGetLastError();
}

}  // namespace flt
