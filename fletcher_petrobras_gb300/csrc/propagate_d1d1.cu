// The step of propagate_fp32.cu in the Der1-Der1 numerics
// (FLETCHER_NUMERICS_D1D1): the floats of the der1der1/ tree
// (der1der1/sample.h:35-120), built without floating-point contraction.
// First derivatives are scaled and kept (pDx = Der1_x(p)/dx,
// pDy = Der1_y(p)/dy) and the mixed derivatives are their first derivatives;
// every operation is rounded on its own in the reference's order, p and q
// separately.
//
// One CTA per SM, persistent, 16 warps of one tile row each.  As
// pxy = Der1_y(pDx) needs pDx of the rows above and below, all warps exchange
// it every plane; lane 0 of the last warp issues the TMA loads (S-2 steps
// ahead) right after its own arrival at that exchange.
#include "device_util.cuh"
#include "fletcher_internal.h"
#include "propagate_fp32_pipe.cuh"
#include "stencil_common.cuh"

namespace flt {

namespace {

template <int TY, int S>
constexpr size_t smem_bytes_d1d1() {
  using G = Geo<TY, true>;
  return size_t(S) * G::STAGE_B + 2 * G::ROW_B + G::AB_B + 8 * S + 8 + 64 + 128;
}

// The producer's position (next step to load), kept in shared memory so it
// costs no registers in the other threads.
struct Cursor {
  Item it;
  int item, k, stage;
};

template <int TY, int S>
__global__ void __launch_bounds__(kTileX *TY, 1)
    k_propagate_d1d1(const __grid_constant__ SingleMaps SM, const __grid_constant__ PropParams P) {
  using G = Geo<TY, true>;
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *smem = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
  f2 *dbuf = reinterpret_cast<f2 *>(smem + S * G::STAGE_B);
  float4 *ABs = reinterpret_cast<float4 *>(smem + S * G::STAGE_B + 2 * G::ROW_B);  // [kABSlots][NT]
  f2 *Cs = reinterpret_cast<f2 *>(ABs + kABSlots * G::NT);                         // [kABSlots][NT]: ch1dxy * pxy
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + S * G::STAGE_B + 2 * G::ROW_B + G::AB_B);
  uint64_t *xchg = full + S;  // pDx rows written (one arrival per warp)
  Cursor *cur = reinterpret_cast<Cursor *>(xchg + 1);

  const int tid = threadIdx.x;
  const int lx = tid & 31;
  const int ly = __shfl_sync(0xffffffffu, tid >> 5, 0);  // warp-uniform
  const int first = P.cta_first[blockIdx.x], end = P.cta_first[blockIdx.x + 1];
  if (first >= end) return;
  const bool producer = tid == (TY - 1) * 32;
  StepMaps maps;
  maps.cur = &SM.cur_halo;
  maps.prev = &SM.prev_pt;
  maps.arr = &SM.arr;
  maps.upd = &SM.upd;
  // Issues the cursor's step into its stage and advances the cursor.
  auto produce = [&]() {
    Cursor c = *cur;
    issue_step<TY>(smem + c.stage * G::STAGE_B, &full[c.stage], c.it, c.k, maps);
    if (++c.stage == S) c.stage = 0;
    if (++c.k >= c.it.z1 + kLag) {
      if (++c.item < end) {
        c.it = decode_item<false>(P.seg[c.item]);
        c.k = c.it.z0 - kRadius;
      }
    }
    *cur = c;
  };
  if (tid == 0) {
    for (int s = 0; s < S; ++s) mbar_init(&full[s], 1);
    mbar_init(xchg, TY);
    mbar_fence_init();
  }
  if (producer) {
    Cursor c;
    c.it = decode_item<false>(P.seg[first]);
    c.item = first;
    c.k = c.it.z0 - kRadius;
    c.stage = 0;
    *cur = c;
  }
  __syncthreads();
  allow_next_launch();
  wait_previous_launch();
  if (producer) {
    tma_prefetch_desc(maps.cur);
    tma_prefetch_desc(maps.prev);
    tma_prefetch_desc(maps.arr);
    tma_prefetch_desc(maps.upd);
    // Prologue: the first S-2 steps of this CTA.
    for (int a = 0; a < S - 2 && cur->item < end; ++a) produce();
  }

  const float sxx = P.inv_dxx, syy = P.inv_dyy, szz = P.inv_dzz;
  const ShotDesc &sd = P.one;
  int stage = 0;
  uint32_t phase = 0, xphase = 0;
  int dsel = 0;
  int abw = 0;  // shared A/B ring slot of the arriving plane (the plane kLag back is at abw + 1)
  for (int item = first; item < end; ++item) {
    const Item it = decode_item<false>(P.seg[item]);
    const int kbeg = it.z0 - kRadius;
    const int kend = it.z1 + kLag;
    const int gx = it.x0 + lx;
    const int gy = it.y0 + ly;
    const int bord = sd.bord, sxs = sd.sx, sys = sd.sy;
    const bool valid = (gx >= bord) && (gx < sxs - bord) && (gy >= bord) && (gy < sys - bord);
    const long plane = (long)sd.pitch * sys;
    unsigned long long *out = reinterpret_cast<unsigned long long *>(sd.F[P.parity ^ 1]) + ((long)gy * sd.pitch + gx);
    const int src_z = sd.src_z, cor_z = sd.cor_z;  // cells are read from `sd` on the (rare) planes
    const int ci = ly * G::TX + lx;
    const int hc = (ly + kRadius) * G::HX + (lx + kRadius);

    f2 Pr[kRing], Dx[kRing], Dy[kRing];

    for (int kb = kbeg; kb < kend; kb += kRing) {
#pragma unroll
      for (int j = 0; j < kRing; ++j) {
        const int k = kb + j;
        if (k >= kend) break;
        unsigned char *st = smem + stage * G::STAGE_B;
        if (!mbar_wait(&full[stage], phase, kWaitLimitNs)) {
          atomicOr(P.err, 1u);
          goto aborted;
        }
        const bool center = (k >= it.z0) && (k < it.z1);
        const bool upd = (k - kLag >= it.z0);
        const bool src_plane = (k == src_z);
        const f2 *H = reinterpret_cast<const f2 *>(st);

        f2 c = H[hc];
        f2 xa[4], xb[4], ya[4], yb[4];
#pragma unroll
        for (int o = 1; o <= 4; ++o) {
          xa[o - 1] = H[hc + o];
          xb[o - 1] = H[hc - o];
          ya[o - 1] = H[hc + o * G::HX];
          yb[o - 1] = H[hc - o * G::HX];
        }
        // Fused source (original/OpenMP/openmp_insertsource.c:7-13): the
        // current p and q gain `src` at the source cell before the update
        // reads them; added to this thread's copies of the plane.
        if (src_plane) {
          const int src_x = sd.src_x, src_y = sd.src_y;
          const f2 sv = splat(P.src);
          f2 dummy;
          if (gy == src_y && abs(src_x - gx) <= kRadius) add_at(c, xa, xb, src_x - gx, sv);
          if (gx == src_x && src_y != gy && abs(src_y - gy) <= kRadius) add_at(dummy, ya, yb, src_y - gy, sv);
        }
        // der1der1/sample.h:35-49: pDx = Der1_x(p) / dx and pDy = Der1_y(p) / dy.
        const f2 d1x = d1_ref(xa[0], xb[0], xa[1], xb[1], xa[2], xb[2], xa[3], xb[3], P.inv_dx);
        const f2 d1y = d1_ref(ya[0], yb[0], ya[1], yb[1], ya[2], yb[2], ya[3], yb[3], P.inv_dy);
        Pr[j] = c;
        Dx[j] = d1x;
        Dy[j] = d1y;
        f2 d2x, d2y;
        f2 *db = dbuf + dsel * (G::HY * G::TX);
        if (center) {
          d2x = d2_ref(c, xa[0], xb[0], xa[1], xb[1], xa[2], xb[2], xa[3], xb[3], sxx);
          d2y = d2_ref(c, ya[0], yb[0], ya[1], yb[1], ya[2], yb[2], ya[3], yb[3], syy);
          // pDx of the tile column and of its 4-row y halo: the row's own
          // value, and warps 0..7 one halo row each (halo-tile rows 0..3 and
          // TY+4..TY+7).
          db[(ly + kRadius) * G::TX + lx] = d1x;
          if (ly < 2 * kRadius) {
            const int hrow = ly < kRadius ? ly : TY + ly;
            const int hb0 = hrow * G::HX + lx + kRadius;
            f2 ha[4], hb[4], dummy;
#pragma unroll
            for (int o = 1; o <= 4; ++o) {
              ha[o - 1] = H[hb0 + o];
              hb[o - 1] = H[hb0 - o];
            }
            if (src_plane && it.y0 - kRadius + hrow == sd.src_y && abs(sd.src_x - gx) <= kRadius)
              add_at(dummy, ha, hb, sd.src_x - gx, splat(P.src));
            db[hrow * G::TX + lx] = d1_ref(ha[0], hb[0], ha[1], hb[1], ha[2], hb[2], ha[3], hb[3], P.inv_dx);
          }
        }
        // Split-phase exchange: announce this warp's pDx (and, by program
        // order, that it has finished the previous step), update plane k-4,
        // which needs no exchanged data, then wait for the other warps.
        __syncwarp();
        if (lx == 0) mbar_arrive(xchg);
        // The producer has passed the exchange of the previous step, so every
        // thread is past the step before it: refill that step's stage with
        // the next step due (S-2 steps ahead of this one).
        if (producer && cur->item < end) {
          fence_proxy_async_smem();
          produce();
        }
        if (upd) {
          const int cs = (j + kRing - kLag) % kRing;  // ring slot of plane k-kLag
          // RP(o): plane k-kLag+o for o = 0..4, k-kLag-(kRing-o) for o > 4.
#define RP(o) Pr[(cs + (o)) % kRing]
#define RX(o) Dx[(cs + (o)) % kRing]
#define RY(o) Dy[(cs + (o)) % kRing]
          constexpr int M1 = kRing - 1, M2 = kRing - 2, M3 = kRing - 3, M4 = kRing - 4;
          // der1der1/sample.h:58-66: pzz, pxz = Der1_z(pDx) / dz, pyz = Der1_z(pDy) / dz.
          const f2 d2z = d2_ref(RP(0), RP(1), RP(M1), RP(2), RP(M2), RP(3), RP(M3), RP(4), RP(M4), szz);
          const f2 dxz = d1_ref(RX(1), RX(M1), RX(2), RX(M2), RX(3), RX(M3), RX(4), RX(M4), P.inv_dz);
          const f2 dyz = d1_ref(RY(1), RY(M1), RY(2), RY(M2), RY(3), RY(M3), RY(4), RY(M4), P.inv_dz);
#undef RP
#undef RX
#undef RY
          const float *cu = reinterpret_cast<const float *>(st + G::OFF_UPD) + (ly * (kUpdateCoef * G::TX) + lx);
          const float czz = cu[0], cxz = cu[G::TX], cyz = cu[2 * G::TX];
          const float v2px = cu[3 * G::TX], v2pz = cu[4 * G::TX];
          const float v2sz = cu[5 * G::TX], v2pn = cu[6 * G::TX];
          const int slot = abw == kLag ? 0 : abw + 1;
          const float4 ab = ABs[slot * G::NT + ci];
          const f2 Ak = mk2(ab.x, ab.y), Bk = mk2(ab.z, ab.w);
          // der1der1/sample.h:70-117 in its order, each operation rounded:
          // h1 = cpxx + cpyy + cpzz + cpxy + cpxz + cpyz (A = cpxx + cpyy,
          // C = cpxy from the plane's arrival), h2 = pxx + pyy + pzz - h1.
          const f2 Ck = Cs[slot * G::NT + ci];
          const f2 h1 = add_rn(add_rn(add_rn(add_rn(Ak, mul_rn(czz, d2z)), Ck), mul_rn(cxz, dxz)), mul_rn(cyz, dyz));
          const f2 h2 = sub_rn(add_rn(Bk, d2z), h1);
          const float h1p = lo(h1), h1q = hi(h1), h2p = lo(h2), h2q = hi(h2);
          const float t = __fmul_rn(v2pz, h1q);
          const float rhsp = __fadd_rn(__fadd_rn(__fmul_rn(v2px, h2p), t), __fmul_rn(v2sz, __fsub_rn(h1p, h1q)));
          const float rhsq = __fsub_rn(__fadd_rn(__fmul_rn(v2pn, h2p), t), __fmul_rn(v2sz, __fsub_rn(h2p, h2q)));
          f2 old = reinterpret_cast<const f2 *>(st + G::OFF_PP)[ci];
          const int zc = k - kLag;
          if (zc == cor_z) {
            if (gx == sd.cor_x && gy == sd.cor_y) old = add2(old, splat(P.cor));
          }
          const f2 now = Pr[cs];
          // pp = 2 pc - pp + rhs * dt * dt (der1der1/sample.h:119-120).
          const f2 nw = add_rn(sub_rn(add_rn(now, now), old), mul_rn(P.dt, mul_rn(P.dt, mk2(rhsp, rhsq))));
          if (valid) out[(long)zc * plane] = nw.v;
        }
        if (!mbar_wait(xchg, xphase, kWaitLimitNs)) {
          // A warp of this CTA stopped arriving (it gave up a wait itself):
          // leave too, so that no thread keeps waiting step after step.
          atomicOr(P.err, 2u);
          goto aborted;
        }
        xphase ^= 1u;
        if (center) {
          // pxy = Der1_y(pDx) / dy (der1der1/sample.h:55); A = cpxx + cpyy,
          // B = pxx + pyy, C = cpxy.
          const f2 *dc = db + (ly + kRadius) * G::TX + lx;
          constexpr int W = G::TX;
          const f2 pxy = d1_ref(dc[W], dc[-W], dc[2 * W], dc[-2 * W], dc[3 * W], dc[-3 * W], dc[4 * W], dc[-4 * W],
                                P.inv_dy);
          const float *ca = reinterpret_cast<const float *>(st + G::OFF_ARR) + (ly * (kArrivalCoef * G::TX) + lx);
          const float cxx = ca[0], cyy = ca[G::TX], cxy = ca[2 * G::TX];
          const f2 av = add_rn(mul_rn(cxx, d2x), mul_rn(cyy, d2y));
          const f2 bv = add_rn(d2x, d2y);
          ABs[abw * G::NT + ci] = make_float4(lo(av), hi(av), lo(bv), hi(bv));
          Cs[abw * G::NT + ci] = mul_rn(cxy, pxy);
        }
        dsel ^= 1;
        abw = abw == kLag ? 0 : abw + 1;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  }
  return;
aborted:
  // A bounded wait gave up.  Every thread leaves (the others give up on
  // their own bounded waits); thread 0 first waits, bounded, for the loads
  // that may still be in flight into this CTA's stages.
  if (tid == 0) {
    for (int a = 0; a < S - 2; ++a) {
      const int s2 = (stage + a) % S;
      (void)mbar_wait(&full[s2], phase ^ uint32_t(stage + a >= S), kWaitLimitNs);
    }
  }
}

}  // namespace

// One shape (kD1D1Rows x kD1D1Stages), single shot.
cudaError_t propagate_d1d1_launch(const PropLaunch &L, cudaStream_t s) {
  constexpr int TY = kD1D1Rows, S = kD1D1Stages;
  constexpr size_t smem = smem_bytes_d1d1<TY, S>();
  static_assert(smem <= 227 * 1024, "Der1-Der1 shape exceeds the shared memory of a CTA");
  static bool ready = false;
  if (!ready) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_propagate_d1d1<TY, S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    ready = true;
  }
  if (L.batch || L.tile_rows != TY || L.stages != S) return cudaErrorInvalidValue;
  return launch_step(k_propagate_d1d1<TY, S>, L.grid, kTileX * TY, smem, s, L.m, L.p);
}

}  // namespace flt
