// The step of propagate_fp32.cu in the Der1-Der1 numerics
// (FLETCHER_NUMERICS_D1D1): the floats of the der1der1/ tree
// (der1der1/sample.h:35-120), built without floating-point contraction.
// First derivatives are scaled and kept (pDx = Der1_x(p)/dx,
// pDy = Der1_y(p)/dy) and the mixed derivatives are their first derivatives;
// every operation is rounded on its own in the reference's order, p and q
// separately.
//
// The warps are specialised as in propagate_fp32.cu: a producer thread issues
// the TMA loads, the halo warps add the step's source and evaluate pDx in the
// tile's 8 halo rows, and 8 compute warps run two tile rows each.  As
// pxy = Der1_y(pDx) needs pDx of the rows above and below, the compute warps
// exchange it every plane: a warp announces its rows, updates plane k-4, which
// needs no exchanged data, and only then waits for the other rows.
//
// What bounds it: the shared-memory pipe and issue.  Against the kernel whose
// compute warps issued the loads and added the source themselves, with p and q
// in scalar instructions: 128 x 112 x 104 updated cells 30.6 -> 26.3 us a step,
// 280 x 200 x 150 170 -> 128, 272^3 327 -> 283; with packed (p, q) instructions
// (mul_rn) 23.9, 118.2 and 252.5, with two cells a thread, as in
// propagate_fp32.cu, 23.5, 117.8 and 248.6.
#include <limits.h>

#include "device_util.cuh"
#include "fletcher_internal.h"
#include "propagate_fp32_pipe.cuh"
#include "stencil_common.cuh"

namespace flt {

namespace {

constexpr int TY = kD1D1Rows, S = kD1D1Stages;
using G = Geo<TY, true>;
constexpr int kHelperWarps = 4, kHaloWarps = kHelperWarps - 1;
constexpr int CW = TY / 2;  // compute warps
constexpr int kThreads = kTileX * (CW + kHelperWarps);
// Registers: 2 x 232 + 32 <= 3 x 168 a sub-partition, as in propagate_fp32.cu.
constexpr int kComputeRegs = 232, kHelperRegs = 32, kLaunchRegs = 168;
static_assert(CW / 4 * kComputeRegs + kHelperWarps / 4 * kHelperRegs <= (CW + kHelperWarps) / 4 * kLaunchRegs,
              "the split exceeds the launch's registers");

// Shared memory: S stages (TMA tiles, pDx of the tile's columns with its
// 4-row halo, a control block), then the in-plane terms (A, B and C) of the
// last 5 planes.
constexpr int OFF_ROWS = G::STAGE_B;
constexpr int OFF_HDR = OFF_ROWS + G::ROW_B;  // the item that starts in the stage
constexpr int OFF_FULL = OFF_HDR + 16;        // barriers: loads landed,
constexpr int OFF_READY = OFF_HDR + 24;       //   source and pDx halo rows written,
constexpr int OFF_XCHG = OFF_HDR + 32;        //   pDx rows of the compute warps written,
constexpr int OFF_EMPTY = OFF_HDR + 40;       //   released by every reader
constexpr int OFF_NZ = OFF_HDR + 64;          // stage 0: -0.0f (mul_rn)
constexpr int SB = OFF_HDR + 128;
constexpr int OFF_ABC = S * SB;  // [kABSlots][A, B, C = ch1dxy * pxy][NT] of 8 bytes
constexpr size_t kSmem = size_t(OFF_ABC) + kABSlots * G::NT * 24 + 128;
static_assert(kSmem <= 227 * 1024, "Der1-Der1 shape exceeds the shared memory of a CTA");
static_assert(OFF_HDR % 128 == 0 && SB % 128 == 0 && OFF_ABC % 128 == 0, "shared-memory alignment");

// HOOK: the fault-injection variant, as in propagate_fp32.cu.
template <bool HOOK>
__global__ void __launch_bounds__(kThreads, 1)
    k_propagate_d1d1(const __grid_constant__ SingleMaps SM, const __grid_constant__ PropParams P) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char *smem = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
  auto bar = [&](unsigned char *st, int off) { return reinterpret_cast<uint64_t *>(st + off); };

  const int tid = threadIdx.x;
  const int lx = tid & 31;
  const int wid = uniform(tid >> 5);
  const int first = P.cta_first[blockIdx.x], nitems = P.cta_first[blockIdx.x + 1] - first;
  if (nitems <= 0) return;
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      unsigned char *st = smem + s * SB;
      mbar_init(bar(st, OFF_FULL), 1);
      mbar_init(bar(st, OFF_READY), kHaloWarps);
      mbar_init(bar(st, OFF_XCHG), CW);
      mbar_init(bar(st, OFF_EMPTY), CW + kHaloWarps);
    }
    mbar_fence_init();
    *reinterpret_cast<volatile float *>(smem + OFF_NZ) = -0.0f;
  }
  __syncthreads();
  allow_next_launch();
  wait_previous_launch();
  // Every wait is bounded.
  auto wait = [&](uint64_t *b, uint32_t parity) { return mbar_spin(b, parity, HOOK ? P.wait_tries : kSpinTries); };
  const ShotDesc &sd = P.one;
  const f2 nz = splat(*reinterpret_cast<volatile float *>(smem + OFF_NZ));

  if (wid >= CW) {
    setmaxnreg_dec<kHelperRegs>();
    const int4 *seg = P.seg + first;
    int stage = 0;
    uint32_t phase = 0;
    if (wid == CW) {
      // ---- producer ----
      if (lx != 0) return;
      StepMaps maps;
      maps.cur = &SM.cur_halo;
      maps.prev = &SM.prev_pt;
      maps.arr = &SM.arr;
      maps.upd = &SM.upd;
      tma_prefetch_desc(maps.cur);
      tma_prefetch_desc(maps.prev);
      tma_prefetch_desc(maps.arr);
      tma_prefetch_desc(maps.upd);
      int4 next = seg[0];
      int issued = 0;
      bool ok = true;
      for (int i = 0; i < nitems && ok; ++i) {
        const int4 w = next;
        const Item it = decode_item<false>(w);
        if (i + 1 < nitems) next = seg[i + 1];
        for (int k = it.z0 - kRadius; k < it.z1 + kLag; ++k) {
          unsigned char *st = smem + stage * SB;
          // (The first S waits pass at once: the stage was never filled.)
          if (!wait(bar(st, OFF_EMPTY), phase ^ 1u)) {
            ok = false;
            break;
          }
          fence_proxy_async_smem();
          if (k == it.z0 - kRadius) *reinterpret_cast<int4 *>(st + OFF_HDR) = w;
          if (!HOOK || issued != P.stall_step || blockIdx.x != 0) issue_step<TY>(st, bar(st, OFF_FULL), it, k, maps);
          ++issued;
          if (++stage == S) {
            stage = 0;
            phase ^= 1u;
          }
        }
      }
      if (!ok) {
        // A bounded wait gave up: wait, bounded, for the loads still in
        // flight, then leave (every other thread gives up on its own waits).
        atomicOr(P.err, 2u);
        for (int a = 1; a <= S && a <= issued; ++a) {
          const int s2 = stage >= a ? stage - a : stage + S - a;
          (void)mbar_wait(bar(smem + s2 * SB, OFF_FULL), stage >= a ? phase : phase ^ 1u, kDrainNs);
        }
      }
      return;
    }
    // ---- halo warps ----
    const int hw = wid - CW - 1;
    const int src_z = sd.src_z;
    auto halo_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * kHaloWarps) : "memory"); };
    [[maybe_unused]] int step = 0;
    int i, k;
    for (i = 0; i < nitems; ++i) {
      const Item it = decode_item<false>(seg[i]);
      for (k = it.z0 - kRadius; k < it.z1 + kLag; ++k) {
        unsigned char *st = smem + stage * SB;
        bool ok = wait(bar(st, OFF_FULL), phase);
        if constexpr (HOOK) ok = ok && !(hw == 1 && blockIdx.x == 0 && step++ == P.quit_step);
        if (!__all_sync(0xffffffffu, ok)) goto gave_up;
        f2 *H = reinterpret_cast<f2 *>(st);
        if (k == src_z) {
          // Fused source (original/OpenMP/openmp_insertsource.c:7-13): the
          // current p and q gain `src` at the source cell before the update
          // reads them.
          const int rx = sd.src_x - (it.x0 - kRadius), ry = sd.src_y - (it.y0 - kRadius);
          if (hw == 0 && lx == 0 && rx >= 0 && rx < G::HX && ry >= 0 && ry < G::HY) {
            H[ry * G::HX + rx] = add2(H[ry * G::HX + rx], splat(P.src));
            fence_proxy_async_smem();
          }
          halo_barrier();
        }
        if (k >= it.z0 && k < it.z1) {
          // pDx of the tile's 4-row y halo (halo-tile rows 0..3 and TY+4..TY+7).
          f2 *db = reinterpret_cast<f2 *>(st + OFF_ROWS);
          for (int r = hw; r < 2 * kRadius; r += kHaloWarps) {
            const int hrow = r < kRadius ? r : TY + r;
            const f2 *h = H + hrow * G::HX + lx + kRadius;
            db[hrow * G::TX + lx] = d1_ref(h[1], h[-1], h[2], h[-2], h[3], h[-3], h[4], h[-4], P.inv_dx, nz);
          }
        }
        __syncwarp();
        if (lx == 0) {
          mbar_arrive(bar(st, OFF_READY));
          mbar_arrive(bar(st, OFF_EMPTY));
        }
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    return;
  gave_up:
    // Meet the other halo warps at every barrier still to come (propagate_fp32.cu).
    if (lx == 0) atomicOr(P.err, 1u);
    for (; i < nitems; ++i, k = INT_MIN) {
      const Item it = decode_item<false>(seg[i]);
      if (src_z >= max(k, it.z0 - kRadius) && src_z < it.z1 + kLag) halo_barrier();
    }
    return;
  }

  // ---- compute warps ----
  setmaxnreg_inc<kComputeRegs>();
  // Lane 16 r + i: cells 2 i and 2 i + 1 of row 2 wid + r.
  const int cx = 2 * (lx & 15);
  const int ly = 2 * wid + (lx >> 4);
  const float sxx = P.inv_dxx, syy = P.inv_dyy, szz = P.inv_dzz;
  const int ci = ly * G::TX + cx;
  const int hc = (ly + kRadius) * G::HX + (cx + kRadius);
  int stage = 0;
  uint32_t phase = 0;
  int abw = 0;  // shared A/B/C ring slot of the arriving plane (the plane kLag back is at abw + 1)
  unsigned char *st = smem;
  for (int item = 0; item < nitems; ++item) {
    if (!wait(bar(st, OFF_READY), phase)) {
      atomicOr(P.err, 1u);
      return;
    }
    const Item it = decode_item<false>(uniform4(*reinterpret_cast<const int4 *>(st + OFF_HDR)));
    const int depth = it.z1 - it.z0;
    const int gx = it.x0 + cx;  // even: a TMA tile starts on 16 bytes
    const int gy = it.y0 + ly;
    const int bord = sd.bord, sxs = sd.sx, sys = sd.sy;
    const bool row = (gy >= bord) && (gy < sys - bord);
    const bool va = row && (gx >= bord) && (gx < sxs - bord);
    const bool vb = row && (gx + 1 >= bord) && (gx + 1 < sxs - bord);
    const long plane = (long)sd.pitch * sys;
    unsigned long long *out =
        reinterpret_cast<unsigned long long *>(sd.F[P.parity ^ 1]) + (it.z0 * plane + (long)gy * sd.pitch + gx);
    // The cell that lacks the last step's source, if it is one of this thread's.
    const int cor_c = sd.cor_x - gx;
    const int cor_k = ((unsigned)cor_c < 2u && gy == sd.cor_y) ? sd.cor_z + kLag - it.z0 : -1000;

    f2 Pr[2][kRing], Dx[2][kRing], Dy[2][kRing];

    for (int kb = -kRadius; kb < depth + kLag; kb += kRing) {
#pragma unroll
      for (int j = 0; j < kRing; ++j) {
        const int k = kb + j;  // plane, counted from the item's first
        if (k >= depth + kLag) break;
        if (!wait(bar(st, OFF_READY), phase)) {
          atomicOr(P.err, 1u);
          return;
        }
        const bool center = (unsigned)k < (unsigned)depth;
        const bool upd = k >= kLag;
        const f2 *H = reinterpret_cast<const f2 *>(st) + hc;
        f2 X[10];           // cells -4 .. +5 of the row
        f2x2 ya[4], yb[4];  // rows +o and -o
#pragma unroll
        for (int o = 0; o < 5; ++o) {
          const f2x2 v = load2(H + 2 * o - 4);
          X[2 * o] = v.a;
          X[2 * o + 1] = v.b;
        }
#pragma unroll
        for (int o = 1; o <= 4; ++o) {
          ya[o - 1] = load2(H + o * G::HX);
          yb[o - 1] = load2(H - o * G::HX);
        }
        // der1der1/sample.h:35-49: pDx = Der1_x(p) / dx and pDy = Der1_y(p) / dy.
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const f2 *x = X + 4 + c;
          Pr[c][j] = x[0];
          Dx[c][j] = d1_ref(x[1], x[-1], x[2], x[-2], x[3], x[-3], x[4], x[-4], P.inv_dx, nz);
        }
        Dy[0][j] = d1_ref(ya[0].a, yb[0].a, ya[1].a, yb[1].a, ya[2].a, yb[2].a, ya[3].a, yb[3].a, P.inv_dy, nz);
        Dy[1][j] = d1_ref(ya[0].b, yb[0].b, ya[1].b, yb[1].b, ya[2].b, yb[2].b, ya[3].b, yb[3].b, P.inv_dy, nz);
        f2 d2x[2], d2y[2];
        f2 *dc = reinterpret_cast<f2 *>(st + OFF_ROWS) + ((ly + kRadius) * G::TX + cx);
        if (center) {
          store2(dc, Dx[0][j], Dx[1][j]);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const f2 *x = X + 4 + c;
            d2x[c] = d2_ref(x[0], x[1], x[-1], x[2], x[-2], x[3], x[-3], x[4], x[-4], sxx, nz);
          }
          d2y[0] = d2_ref(X[4], ya[0].a, yb[0].a, ya[1].a, yb[1].a, ya[2].a, yb[2].a, ya[3].a, yb[3].a, syy, nz);
          d2y[1] = d2_ref(X[5], ya[0].b, yb[0].b, ya[1].b, yb[1].b, ya[2].b, yb[2].b, ya[3].b, yb[3].b, syy, nz);
        }
        // Split-phase exchange: announce this warp's pDx, update plane k-4,
        // then wait for the other rows.
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, OFF_XCHG));
        if (upd) {
          const int cs = (j + kRing - kLag) % kRing;  // ring slot of plane k-kLag
          constexpr int M1 = kRing - 1, M2 = kRing - 2, M3 = kRing - 3, M4 = kRing - 4;
          const float *cu = reinterpret_cast<const float *>(st + G::OFF_UPD) + (ly * (kUpdateCoef * G::TX) + cx);
          auto pair = [&](int t) { return *reinterpret_cast<const float2 *>(cu + t * G::TX); };
          const float2 czz = pair(0), cxz = pair(1), cyz = pair(2);
          const float2 v2px = pair(3), v2pz = pair(4), v2sz = pair(5), v2pn = pair(6);
          const f2 *ab = reinterpret_cast<const f2 *>(smem + OFF_ABC) + (abw == kLag ? 0 : abw + 1) * (3 * G::NT) + ci;
          const f2x2 A = load2(ab), Bv = load2(ab + G::NT), C = load2(ab + 2 * G::NT);
          f2x2 old = load2(reinterpret_cast<const f2 *>(st + G::OFF_PP) + ci);
          if (k == cor_k) {
            if (cor_c == 0) old.a = add2(old.a, splat(P.cor));
            else old.b = add2(old.b, splat(P.cor));
          }
          f2 nw[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            auto of = [&](float2 v) { return c ? v.y : v.x; };
            // RP(o): plane k-kLag+o for o = 0..4, k-kLag-(kRing-o) for o > 4.
#define RP(o) Pr[c][(cs + (o)) % kRing]
#define RX(o) Dx[c][(cs + (o)) % kRing]
#define RY(o) Dy[c][(cs + (o)) % kRing]
            // der1der1/sample.h:58-66: pzz, pxz = Der1_z(pDx) / dz, pyz = Der1_z(pDy) / dz.
            const f2 d2z = d2_ref(RP(0), RP(1), RP(M1), RP(2), RP(M2), RP(3), RP(M3), RP(4), RP(M4), szz, nz);
            const f2 dxz = d1_ref(RX(1), RX(M1), RX(2), RX(M2), RX(3), RX(M3), RX(4), RX(M4), P.inv_dz, nz);
            const f2 dyz = d1_ref(RY(1), RY(M1), RY(2), RY(M2), RY(3), RY(M3), RY(4), RY(M4), P.inv_dz, nz);
#undef RP
#undef RX
#undef RY
            // der1der1/sample.h:70-117 in its order, each operation rounded:
            // h1 = cpxx + cpyy + cpzz + cpxy + cpxz + cpyz (A = cpxx + cpyy,
            // C = cpxy from the plane's arrival), h2 = pxx + pyy + pzz - h1.
            const f2 h1 = add2(add2(add2(add2(c ? A.b : A.a, mul_rn(of(czz), d2z, nz)), c ? C.b : C.a),
                                    mul_rn(of(cxz), dxz, nz)),
                               mul_rn(of(cyz), dyz, nz));
            const f2 h2 = sub2(add2(c ? Bv.b : Bv.a, d2z), h1);
            const float h1p = lo(h1), h1q = hi(h1), h2p = lo(h2), h2q = hi(h2);
            const float t = __fmul_rn(of(v2pz), h1q);
            const float rhsp = __fadd_rn(__fadd_rn(__fmul_rn(of(v2px), h2p), t), __fmul_rn(of(v2sz), __fsub_rn(h1p, h1q)));
            const float rhsq = __fsub_rn(__fadd_rn(__fmul_rn(of(v2pn), h2p), t), __fmul_rn(of(v2sz), __fsub_rn(h2p, h2q)));
            const f2 now = Pr[c][cs];
            // pp = 2 pc - pp + rhs * dt * dt (der1der1/sample.h:119-120).
            nw[c] = add2(sub2(add2(now, now), c ? old.b : old.a),
                         mul_rn(P.dt, mul_rn(P.dt, mk2(rhsp, rhsq), nz), nz));
          }
          if (va && vb) {
            *reinterpret_cast<ulonglong2 *>(out) = make_ulonglong2(nw[0].v, nw[1].v);
          } else {
            if (va) out[0] = nw[0].v;
            if (vb) out[1] = nw[1].v;
          }
          out += plane;
        }
        if (center) {
          if (!wait(bar(st, OFF_XCHG), phase)) {
            atomicOr(P.err, 2u);
            return;
          }
          // pxy = Der1_y(pDx) / dy (der1der1/sample.h:55); A = cpxx + cpyy,
          // B = pxx + pyy, C = cpxy.
          f2x2 ra[4], rb[4];
#pragma unroll
          for (int o = 1; o <= 4; ++o) {
            ra[o - 1] = load2(dc + o * G::TX);
            rb[o - 1] = load2(dc - o * G::TX);
          }
          const f2 pxy[2] = {
              d1_ref(ra[0].a, rb[0].a, ra[1].a, rb[1].a, ra[2].a, rb[2].a, ra[3].a, rb[3].a, P.inv_dy, nz),
              d1_ref(ra[0].b, rb[0].b, ra[1].b, rb[1].b, ra[2].b, rb[2].b, ra[3].b, rb[3].b, P.inv_dy, nz)};
          const float *ca = reinterpret_cast<const float *>(st + G::OFF_ARR) + (ly * (kArrivalCoef * G::TX) + cx);
          auto pair = [&](int t) { return *reinterpret_cast<const float2 *>(ca + t * G::TX); };
          const float2 cxx = pair(0), cyy = pair(1), cxy = pair(2);
          f2 *ab = reinterpret_cast<f2 *>(smem + OFF_ABC) + abw * (3 * G::NT) + ci;
          store2(ab, add2(mul_rn(cxx.x, d2x[0], nz), mul_rn(cyy.x, d2y[0], nz)),
                 add2(mul_rn(cxx.y, d2x[1], nz), mul_rn(cyy.y, d2y[1], nz)));
          store2(ab + G::NT, add2(d2x[0], d2y[0]), add2(d2x[1], d2y[1]));
          store2(ab + 2 * G::NT, mul_rn(cxy.x, pxy[0], nz), mul_rn(cxy.y, pxy[1], nz));
        }
        // This warp is done with the stage.
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, OFF_EMPTY));
        abw = abw == kLag ? 0 : abw + 1;
        st = stage == S - 1 ? smem : st + SB;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  }
}

}  // namespace

template <bool HOOK>
static cudaError_t launch_d1d1(const PropLaunch &L, cudaStream_t s) {
  static bool ready = false;
  if (!ready) {
    const cudaError_t e = prepare_step_kernel((const void *)k_propagate_d1d1<HOOK>, kSmem, kLaunchRegs);
    if (e != cudaSuccess) return e;
    ready = true;
  }
  return launch_step(k_propagate_d1d1<HOOK>, L.grid, kThreads, kSmem, s, L.m, L.p);
}

// One shape (kD1D1Rows x kD1D1Stages), single shot.
cudaError_t propagate_d1d1_launch(const PropLaunch &L, cudaStream_t s) {
  if (L.batch || L.tile_rows != TY || L.stages != S) return cudaErrorInvalidValue;
  return fault_injected(L.p) ? launch_d1d1<true>(L, s) : launch_d1d1<false>(L, s);
}

}  // namespace flt
