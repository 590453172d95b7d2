// Plain FP32 Fletcher TTI step for sm_103a.
//
// Computes, for every cell of [bord, s-bord)^3, the coupled p/q update of
// original/sample.h:32-89 (Der2 / DerCross of original/derivatives.h:37-68,
// weighted by the ch1d** and v2** coefficients of original/precomp.h), with
// the source of original/OpenMP/openmp_insertsource.c:7-13 fused in.
//
// Structure (one CTA per SM, persistent, warp-specialised):
//  * a work item is a 32 x TY column tile of one z range; the CTA streams its
//    planes k = z0-4 .. z1+3 in z through a ring of S shared-memory stages;
//  * the producer (one thread of the helper warps) issues a stage's TMA
//    loads as soon as every reader has released it: the (p,q) halo tile of
//    plane k (box 40 x (TY+8)), the three in-plane coefficients of plane k,
//    and the seven other coefficients and the previous (p,q) of plane k-4,
//    which is updated at this step;
//  * the halo warps (three helper warps) evaluate D1y in the tile's 8 halo
//    columns, ahead of the compute warps, and add the step's source to the
//    tile of the plane that holds it;
//  * TY / 2 compute warps, each two rows: a thread owns the columns of two
//    cells that lie side by side in x.  When plane k arrives it reads its 9-point
//    x and y neighbourhoods from shared memory, 16 bytes at a time, and forms
//    Der2x, Der2y and the first derivatives D1x, D1y; DerCross xy
//    is D1x applied to D1y, whose rows of the tile only this warp and the
//    halo columns write (so compute warps never wait for one another);
//    DerCross xz and yz are the z first derivative of the D1x / D1y values,
//    which each thread keeps for 9 planes in registers, as it keeps p and q
//    for Der2z; the in-plane terms A and B wait in shared memory;
//  * both fields travel as one 64-bit (p, q) pair and are updated with the
//    packed .f32x2 add/mul/fma instructions;
//  * plane k-4 is completed at step k and written with coalesced 128-bit
//    stores into the previous-field buffer (in place).
//
// What bounds it: HBM where the grid is large, elsewhere the latency of a warp's
// plane (two or three warps a scheduler: half of its issue slots and 45 to 70%
// of the shared-memory pipe are used).  At 504^3 (183 M updated cells, 64 B each)
// a step takes 1.76 to 1.79 ms, 97 to 98% of the measured copy bandwidth; a
// plane of a tile alone on the GPU takes an SM 0.60 us.  Before the warps were
// specialised, 16 warps that exchanged D1y, and refilled the stages, in one
// CTA-wide exchange a plane took 2.22 ms.  What made the difference:
//  * the loop is unrolled over the 9 ring slots, and with the producer, the
//    source and the timed waits in it the code was 102 KB (the instruction
//    fetch was the stall of 1.1 of 8.4 cycles an issue); moved to the helper
//    warps and counted waits, it is 50 KB.  (One loop body with a switch over
//    the slots, 24 KB, is slower: the loads of a plane no longer overlap its
//    arithmetic; 272^3 updated cells 199 -> 215 us.);
//  * a stage is refilled the moment its last reader releases it, whichever
//    warp that is, and the warps may run up to S planes apart.  (Groups of 4
//    warps that exchange among themselves, with the refill still issued by
//    a compute warp, took 2.48 ms: warps that run ahead of the producing
//    warp find their loads not yet issued.)
//  * one wait a step (for the halo warps, which wait for the loads) and one
//    base address for all that a stage holds: 14% fewer instructions, 272^3
//    updated cells 205.1 -> 203.5 us;
//  * two cells a thread share a window of 10 cells instead of two of 9, read
//    as five 16-byte words: 72 instead of 88 shared-memory wavefronts a row
//    and 26% fewer instructions than one cell a thread.  In us a step: media
//    table 192^3 updated cells 69.7 -> 63.3, 150 x 97 x 260 49.5 -> 45.2, 88^3
//    12.4 -> 11.7, 312^3 302.2 -> 298.7, 272^3 200.2 -> 199.4; 504^3 1760 -> 1765 and
//    a 36 x 32 x 28 grid 5.5 -> 5.65 (fewer warps for one plane's latency).  With
//    A and B in registers too the loads lose their overlap (272^3 212 us, with
//    A alone 206).
// 16 rows: 8 compute warps at 232 registers hold the 54 ring values and a
// plane's neighbourhood without a spill; 12 rows take 81 and 8 rows (two
// CTAs an SM) 76 us where 16 rows take 73.3 (192^3 updated cells).
//
// Media-table layout (template parameter MT): instead of the ten coefficient
// planes a stage holds the one-byte medium ids of planes k and k-4 and the
// four velocity terms of plane k-4; the six angle terms come from a table
// of at most 256 media loaded into shared memory once per launch.  The
// floats read are the same as in the plane layout, so results are
// bit-identical; the stream drops from 64 to 41 bytes per cell.
//
// DerCross(p, a, b) equals D1_b(D1_a(p)) exactly in real arithmetic because
// its weights are the products L_i L_j of the first-derivative weights
// (original/derivatives.h:13-31); the FP32 rounding differs from the
// reference's grouped sum, which the parity tolerance covers.
#include <limits.h>

#include "device_util.cuh"
#include "fletcher_internal.h"
#include "propagate_fp32_pipe.cuh"
#include "stencil_common.cuh"

namespace flt {

constexpr int kHelperWarps = 4;  // producer warp + 3 halo warps: one warpgroup (setmaxnreg works on warpgroups)
constexpr int kHaloWarps = kHelperWarps - 1;

// Shared memory of a CTA: S stages, then what is not per stage.  A stage
// holds its TMA tiles (Geo), the D1y exchange rows of its plane, the in-plane
// terms (A, B) of its plane when five stages match their five slots, and a
// control block: everything a step addresses is one base away.  (The 8 x 5
// shape, whose two CTAs share an SM's memory, has two exchange buffers.)
template <int TY, int S, bool MT>
struct Layout {
  using G = Geo<TY, false, MT>;
  static constexpr int NB = (TY <= 8 && S > 4) ? 2 : S;
  static constexpr bool ROWS_IN = NB == S, AB_IN = S == kABSlots;
  static constexpr int AB_SLOT = G::NT * 16;
  static constexpr int OFF_SROWS = G::STAGE_B;
  static constexpr int OFF_SAB = OFF_SROWS + (ROWS_IN ? G::ROW_B : 0);
  static constexpr int OFF_CTL = OFF_SAB + (AB_IN ? AB_SLOT : 0);
  static constexpr int OFF_HDR = OFF_CTL;         // the item that starts in the stage
  static constexpr int OFF_FULL = OFF_CTL + 16;   // barriers: loads landed,
  static constexpr int OFF_READY = OFF_CTL + 24;  //   halo columns and source written too,
  static constexpr int OFF_EMPTY = OFF_CTL + 32;  //   released by every reader
  static constexpr int SB = OFF_CTL + 128;
  static constexpr int OFF_ROWS = S * SB;  // [NB] exchange buffers, when not in the stages
  static constexpr int OFF_AB = OFF_ROWS + (ROWS_IN ? 0 : NB * G::ROW_B);
  static constexpr int OFF_TAB = OFF_AB + (AB_IN ? 0 : kABSlots * AB_SLOT);
  static constexpr size_t BYTES = size_t(OFF_TAB) + G::TAB_B + 128;
  static_assert(OFF_CTL % 128 == 0 && OFF_ROWS % 128 == 0 && OFF_AB % 128 == 0 && OFF_TAB % 128 == 0,
                "shared-memory alignment");
};

// Register split (setmaxnreg): the compute warps take what the helper warps
// give back.  Per SM sub-partition, two compute warps (8 rows: one) and one
// helper warp share the launch's registers, 168 a thread (8 rows: 128):
// 2 x 232 + 32 <= 3 x 168, 224 + 32 = 2 x 128.
constexpr int kHelperRegs = 32;
template <int TY>
struct Regs {
  static constexpr int kWarps = (TY / 2 + 3) / 4 * 4;  // compute warps, whole warpgroups (12 rows leave two idle)
  static constexpr int kCompute = TY == 8 ? 224 : 232;
  static constexpr int kLaunch = TY == 8 ? 128 : 168;
  static_assert((kWarps / 4) * kCompute + kHelperRegs <= (kWarps / 4 + 1) * kLaunch,
                "the split exceeds the launch's registers");
};

// HOOK: the fault-injection variant (waits limited to P.wait_tries tries, CTA 0
// skipping the loads of its P.stall_step-th step, or one of its halo warps
// giving up at its P.quit_step-th), launched only when a test injects a fault.  MT: the media-table layout of the coefficients.
template <int TY, int S, bool ISO, bool BATCH, int MINB, bool HOOK = false, bool MT = false>
__global__ void __launch_bounds__(kTileX *(Regs<TY>::kWarps + kHelperWarps), MINB)
    k_propagate_fp32(const __grid_constant__ SingleMaps SM, const __grid_constant__ PropParams P) {
  static_assert(!MT || (!BATCH && !HOOK), "the media-table layout runs single-shot plain steps");
  using G = Geo<TY, false, MT>;
  using L = Layout<TY, S, MT>;
  extern __shared__ unsigned char smem_dyn[];
  // Align in the shared window (pointer arithmetic on the shared array keeps
  // every access below a shared-memory access).
  unsigned char *smem = smem_dyn + ((128u - (smem_addr(smem_dyn) & 127u)) & 127u);
  float *s_med = reinterpret_cast<float *>(smem + L::OFF_TAB);  // [6][256] (MT)
  auto bar = [&](unsigned char *st, int off) { return reinterpret_cast<uint64_t *>(st + off); };

  const int tid = threadIdx.x;
  const int lx = tid & 31;
  const int wid = uniform(tid >> 5);
  constexpr int CW = Regs<TY>::kWarps;
  const int first = P.cta_first[blockIdx.x], nitems = P.cta_first[blockIdx.x + 1] - first;
  if (nitems <= 0) return;
  constexpr int kHalo = TY / 4 < kHaloWarps ? TY / 4 : kHaloWarps;  // halo warps with work
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      unsigned char *st = smem + s * L::SB;
      mbar_init(bar(st, L::OFF_FULL), 1);
      mbar_init(bar(st, L::OFF_READY), kHalo);
      mbar_init(bar(st, L::OFF_EMPTY), TY / 2 + kHalo);
    }
    mbar_fence_init();
  }
  if constexpr (MT) {
    for (int i = tid; i < kAngleCoef * kMediaMax; i += kTileX * (CW + kHelperWarps)) s_med[i] = P.media[i];
  }
  __syncthreads();
  allow_next_launch();
  wait_previous_launch();
  // Every wait is bounded.
  auto wait = [&](uint64_t *b, uint32_t parity) { return mbar_spin(b, parity, HOOK ? P.wait_tries : kSpinTries); };

  if (wid >= CW) {
    setmaxnreg_dec<kHelperRegs>();
    const int4 *seg = P.seg + first;
    int stage = 0;
    uint32_t phase = 0;
    if (wid == CW) {
      // ---- producer ----
      if (lx != 0) return;
      auto maps_of = [&](int shot) {
        StepMaps m;
        if constexpr (BATCH) {
          const ShotMaps *sm = P.maps + shot;
          m.cur = &sm->halo[P.parity];
          m.prev = &sm->pt[P.parity ^ 1];
          m.arr = &sm->arr;
          m.upd = &sm->upd;
        } else {
          m.cur = &SM.cur_halo;
          m.prev = &SM.prev_pt;
          m.arr = &SM.arr;
          m.upd = &SM.upd;
        }
        m.ids = &SM.ids;
        m.vel = &SM.vel;
        return m;
      };
      auto prefetch = [&](int shot) {
        const StepMaps m = maps_of(shot);
        tma_prefetch_desc(m.cur);
        tma_prefetch_desc(m.prev);
        tma_prefetch_desc(MT ? m.ids : m.arr);
        tma_prefetch_desc(MT ? m.vel : m.upd);
      };
      int4 next = seg[0];
      prefetch(decode_item<BATCH>(next).shot);
      int issued = 0;
      bool ok = true;
      for (int i = 0; i < nitems && ok; ++i) {
        const int4 w = next;
        const Item it = decode_item<BATCH>(w);
        if (i + 1 < nitems) {
          next = seg[i + 1];
          // Batched shots keep their tensor maps in global memory: fetch the
          // next item's into the descriptor cache an item ahead.
          if constexpr (BATCH) prefetch(decode_item<BATCH>(next).shot);
        }
        const StepMaps m = maps_of(it.shot);
        for (int k = it.z0 - kRadius; k < it.z1 + kLag; ++k) {
          // (The first S waits pass at once: the stage was never filled.)
          unsigned char *st = smem + stage * L::SB;
          if (!wait(bar(st, L::OFF_EMPTY), phase ^ 1u)) {
            ok = false;
            break;
          }
          fence_proxy_async_smem();
          if (k == it.z0 - kRadius) *reinterpret_cast<int4 *>(st + L::OFF_HDR) = w;
          // Test hook: CTA 0 skips the loads of its P.stall_step-th step, so
          // that the waits for that stage give up.
          if (!HOOK || issued != P.stall_step || blockIdx.x != 0)
            issue_step<TY, MT>(st, bar(st, L::OFF_FULL), it, k, m);
          ++issued;
          if (++stage == S) {
            stage = 0;
            phase ^= 1u;
          }
        }
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
    // ---- halo warps ----
    const int hw = wid - CW - 1;
    if (hw >= kHalo) return;
    const int hxc = (lx & 7) < 4 ? (lx & 7) : G::TX + (lx & 7);  // lane -> halo column, row lane / 8 of a group of 4
    [[maybe_unused]] int step = 0;
    auto halo_barrier = [] { asm volatile("bar.sync 1, %0;" ::"n"(32 * kHalo) : "memory"); };
    int rb = 0;
    int i, k;
    for (i = 0; i < nitems; ++i) {
      const Item it = decode_item<BATCH>(seg[i]);
      const ShotDesc &sd = BATCH ? P.shots[it.shot] : P.one;
      const int src_z = sd.src_z;
      for (k = it.z0 - kRadius; k < it.z1 + kLag; ++k) {
        unsigned char *st = smem + stage * L::SB;
        bool ok = wait(bar(st, L::OFF_FULL), phase);
        if constexpr (L::NB < S) {
          // The row buffer's last readers: the step NB back.
          const int es = stage >= L::NB ? stage - L::NB : stage + S - L::NB;
          ok = ok && wait(bar(smem + es * L::SB, L::OFF_EMPTY), stage >= L::NB ? phase : phase ^ 1u);
        }
        // Test hook: a halo warp of CTA 0 gives up at its P.quit_step-th step.
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
          f2 *db = reinterpret_cast<f2 *>(L::ROWS_IN ? st + L::OFF_SROWS : smem + L::OFF_ROWS + rb * G::ROW_B);
          for (int r = hw * 4 + (lx >> 3); r < TY; r += 4 * kHalo) {
            const f2 *h = H + (r + kRadius) * G::HX + hxc;
            f2 d = mul2(splat(cL1), sub2(h[G::HX], h[-G::HX]));
            d = fma2(splat(cL2), sub2(h[2 * G::HX], h[-2 * G::HX]), d);
            d = fma2(splat(cL3), sub2(h[3 * G::HX], h[-3 * G::HX]), d);
            d = fma2(splat(cL4), sub2(h[4 * G::HX], h[-4 * G::HX]), d);
            db[r * G::HX + hxc] = d;
          }
        }
        __syncwarp();
        if (lx == 0) {
          mbar_arrive(bar(st, L::OFF_READY));
          mbar_arrive(bar(st, L::OFF_EMPTY));
        }
        if (!L::ROWS_IN && ++rb == L::NB) rb = 0;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
    return;
  gave_up:
    // Another halo warp's wait may have succeeded: this one meets the others at
    // every barrier still to come before it leaves, so that none waits there for
    // a warp that has left.  (Inside the loop this code costs the media-table
    // layout 1%.)
    if (lx == 0) atomicOr(P.err, 1u);
    for (; i < nitems; ++i, k = INT_MIN) {
      const Item it = decode_item<BATCH>(seg[i]);
      const int src_z = (BATCH ? P.shots[it.shot] : P.one).src_z;
      if (src_z >= max(k, it.z0 - kRadius) && src_z < it.z1 + kLag) halo_barrier();
    }
    return;
  }

  // ---- compute warps ----
  setmaxnreg_inc<Regs<TY>::kCompute>();
  if (wid >= TY / 2) return;
  // Lane 16 r + i: cells 2 i and 2 i + 1 of row 2 wid + r.
  const int cx = 2 * (lx & 15);
  const int ly = 2 * wid + (lx >> 4);
  // Spacing factors (unused on isotropic grids).
  const float sxy = P.inv_dxy, sxz = P.inv_dxz, syz = P.inv_dyz;
  const float sxx = P.inv_dxx, syy = P.inv_dyy, szz = P.inv_dzz;
  const int ci = ly * G::TX + cx;
  const int hc = (ly + kRadius) * G::HX + (cx + kRadius);
  int stage = 0;
  uint32_t phase = 0;
  int rb = 0;   // exchange buffer (when not in the stages)
  int abw = 0;  // shared A/B ring slot of the arriving plane (the plane kLag back is at abw + 1)
  unsigned char *st = smem;
  for (int item = 0; item < nitems; ++item) {
    if (!wait(bar(st, L::OFF_READY), phase)) {
      atomicOr(P.err, 1u);
      return;
    }
    const Item it = decode_item<BATCH>(uniform4(*reinterpret_cast<const int4 *>(st + L::OFF_HDR)));
    const ShotDesc &sd = BATCH ? P.shots[it.shot] : P.one;
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

    const int y0w = it.y0 + 2 * wid;
    if (P.skip_rows && (y0w + 1 < bord || y0w >= sys - bord)) {
      // Two rows outside the updated region: nothing to compute, only the
      // stages to release in step.  (Not where the plan deals every tile
      // alike: tiles that run ahead of their neighbours share fewer halo
      // rows; 312^3 updated cells 304.7 -> 308.5 us.)
      for (int k = -kRadius; k < depth + kLag; ++k) {
        if (!wait(bar(st, L::OFF_READY), phase)) {
          atomicOr(P.err, 1u);
          return;
        }
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, L::OFF_EMPTY));
        if (!L::AB_IN) abw = abw == kLag ? 0 : abw + 1;
        if (!L::ROWS_IN && ++rb == L::NB) rb = 0;
        st = stage == S - 1 ? smem : st + L::SB;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
      continue;
    }

    f2 Pr[2][kRing], Dx[2][kRing], Dy[2][kRing];

    for (int kb = -kRadius; kb < depth + kLag; kb += kRing) {
#pragma unroll
      for (int j = 0; j < kRing; ++j) {
        const int k = kb + j;  // plane, counted from the item's first
        if (k >= depth + kLag) break;
        if (!wait(bar(st, L::OFF_READY), phase)) {
          atomicOr(P.err, 1u);
          return;
        }
        unsigned char *const st_next = stage == S - 1 ? smem : st + L::SB;
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
        f2 d2x[2], d2y[2];
        f2 *dr = reinterpret_cast<f2 *>(L::ROWS_IN ? st + L::OFF_SROWS : smem + L::OFF_ROWS + rb * G::ROW_B) +
                 (ly * G::HX + cx + kRadius);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const f2 *x = X + 4 + c;
          Pr[c][j] = x[0];
          Dx[c][j] = d1(x[1], x[-1], x[2], x[-2], x[3], x[-3], x[4], x[-4]);
        }
        Dy[0][j] = d1(ya[0].a, yb[0].a, ya[1].a, yb[1].a, ya[2].a, yb[2].a, ya[3].a, yb[3].a);
        Dy[1][j] = d1(ya[0].b, yb[0].b, ya[1].b, yb[1].b, ya[2].b, yb[2].b, ya[3].b, yb[3].b);
        if (center) {
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const f2 *x = X + 4 + c;
            d2x[c] = scale<ISO>(d2(x[0], x[1], x[-1], x[2], x[-2], x[3], x[-3], x[4], x[-4]), sxx);
          }
          d2y[0] = scale<ISO>(d2(X[4], ya[0].a, yb[0].a, ya[1].a, yb[1].a, ya[2].a, yb[2].a, ya[3].a, yb[3].a), syy);
          d2y[1] = scale<ISO>(d2(X[5], ya[0].b, yb[0].b, ya[1].b, yb[1].b, ya[2].b, yb[2].b, ya[3].b, yb[3].b), syy);
          store2(dr, Dy[0][j], Dy[1][j]);
        }
        __syncwarp();
        if (upd) {
          const int cs = (j + kRing - kLag) % kRing;  // ring slot of plane k-kLag
          constexpr int M1 = kRing - 1, M2 = kRing - 2, M3 = kRing - 3, M4 = kRing - 4;
          const float *cu =
              reinterpret_cast<const float *>(st + G::OFF_UPD) + (ly * ((MT ? kVelCoef : kUpdateCoef) * G::TX) + cx);
          float2 czz, cxz, cyz, v2px, v2pz, v2sz, v2pn;
          auto pair = [](const float *p) { return *reinterpret_cast<const float2 *>(p); };
          if constexpr (MT) {
            const uchar2 md = *reinterpret_cast<const uchar2 *>(st + G::OFF_IDU + ci);
            auto term = [&](int t) { return make_float2(s_med[t * kMediaMax + md.x], s_med[t * kMediaMax + md.y]); };
            czz = term(DC_ZZ);
            cxz = term(DC_XZ);
            cyz = term(DC_YZ);
            v2px = pair(cu);
            v2pz = pair(cu + G::TX);
            v2sz = pair(cu + 2 * G::TX);
            v2pn = pair(cu + 3 * G::TX);
          } else {
            czz = pair(cu);
            cxz = pair(cu + G::TX);
            cyz = pair(cu + 2 * G::TX);
            v2px = pair(cu + 3 * G::TX);
            v2pz = pair(cu + 4 * G::TX);
            v2sz = pair(cu + 5 * G::TX);
            v2pn = pair(cu + 6 * G::TX);
          }
          // (With five slots the plane kLag back is the next one round.)
          const f2 *ab = reinterpret_cast<const f2 *>(
              L::AB_IN ? st_next + L::OFF_SAB : smem + L::OFF_AB + (abw == kLag ? 0 : abw + 1) * L::AB_SLOT);
          const f2x2 A = load2(ab + ci), Bv = load2(ab + G::NT + ci);
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
            const f2 d2z = scale<ISO>(d2(RP(0), RP(1), RP(M1), RP(2), RP(M2), RP(3), RP(M3), RP(4), RP(M4)), szz);
            const f2 dxz = scale<ISO>(d1(RX(1), RX(M1), RX(2), RX(M2), RX(3), RX(M3), RX(4), RX(M4)), sxz);
            const f2 dyz = scale<ISO>(d1(RY(1), RY(M1), RY(2), RY(M2), RY(3), RY(M3), RY(4), RY(M4)), syz);
#undef RP
#undef RX
#undef RY
            const f2 h1 = fma2(splat(of(cyz)), dyz,
                               fma2(splat(of(cxz)), dxz, fma2(splat(of(czz)), d2z, c ? A.b : A.a)));
            const f2 h2 = sub2(add2(c ? Bv.b : Bv.a, d2z), h1);
            const float h1p = lo(h1), h1q = hi(h1), h2p = lo(h2), h2q = hi(h2);
            // Explicit roundings: every unrolled copy computes identical floats.
            const float t = __fmul_rn(of(v2pz), h1q);
            const float rhsp = __fmaf_rn(of(v2sz), __fsub_rn(h1p, h1q), __fmaf_rn(of(v2px), h2p, t));
            const float rhsq = __fmaf_rn(-of(v2sz), __fsub_rn(h2p, h2q), __fmaf_rn(of(v2pn), h2p, t));
            const f2 cur = Pr[c][cs];
            nw[c] = fma2(mk2(rhsp, rhsq), splat(P.dt2), sub2(add2(cur, cur), c ? old.b : old.a));
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
          f2 Y[10];  // D1y of cells -4 .. +5 of the row
#pragma unroll
          for (int o = 0; o < 5; ++o) {
            if (o == 2) continue;
            const f2x2 v = load2(dr + 2 * o - 4);
            Y[2 * o] = v.a;
            Y[2 * o + 1] = v.b;
          }
          Y[4] = Dy[0][j];
          Y[5] = Dy[1][j];
          float2 cxx, cyy, cxy;
          if constexpr (MT) {
            const uchar2 md = *reinterpret_cast<const uchar2 *>(st + G::OFF_IDC + ci);
            auto term = [&](int t) { return make_float2(s_med[t * kMediaMax + md.x], s_med[t * kMediaMax + md.y]); };
            cxx = term(DC_XX);
            cyy = term(DC_YY);
            cxy = term(DC_XY);
          } else {
            const float *ca = reinterpret_cast<const float *>(st + G::OFF_ARR) + (ly * (kArrivalCoef * G::TX) + cx);
            cxx = *reinterpret_cast<const float2 *>(ca);
            cyy = *reinterpret_cast<const float2 *>(ca + G::TX);
            cxy = *reinterpret_cast<const float2 *>(ca + 2 * G::TX);
          }
          f2 av[2], bv[2];
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            auto of = [&](float2 v) { return c ? v.y : v.x; };
            const f2 *y = Y + 4 + c;
            const f2 dxy = scale<ISO>(d1(y[1], y[-1], y[2], y[-2], y[3], y[-3], y[4], y[-4]), sxy);
            av[c] = fma2(splat(of(cxy)), dxy, fma2(splat(of(cyy)), d2y[c], mul2(splat(of(cxx)), d2x[c])));
            bv[c] = add2(d2x[c], d2y[c]);
          }
          f2 *ab = reinterpret_cast<f2 *>(L::AB_IN ? st + L::OFF_SAB : smem + L::OFF_AB + abw * L::AB_SLOT);
          store2(ab + ci, av[0], av[1]);
          store2(ab + G::NT + ci, bv[0], bv[1]);
        }
        // This warp is done with the stage.
        __syncwarp();
        if (lx == 0) mbar_arrive(bar(st, L::OFF_EMPTY));
        if (!L::AB_IN) abw = abw == kLag ? 0 : abw + 1;
        if (!L::ROWS_IN && ++rb == L::NB) rb = 0;
        st = st_next;
        if (++stage == S) {
          stage = 0;
          phase ^= 1u;
        }
      }
    }
  }
}

// ---- host side ---------------------------------------------------------------

template <int TY, int S, bool MT = false>
constexpr size_t smem_bytes() {
  return Layout<TY, S, MT>::BYTES;
}

template <int TY, int S, int MINB>
static cudaError_t prepare_t() {
  constexpr size_t smem = smem_bytes<TY, S>();
  static_assert(smem * MINB + MINB * 1024 <= 228 * 1024, "tile shape exceeds the shared memory of an SM");
  cudaError_t e = cudaSuccess;
  for (auto kern : {k_propagate_fp32<TY, S, true, false, MINB>, k_propagate_fp32<TY, S, false, false, MINB>,
                    k_propagate_fp32<TY, S, true, true, MINB>, k_propagate_fp32<TY, S, false, true, MINB>})
    if (e == cudaSuccess) e = prepare_step_kernel((const void *)kern, smem, Regs<TY>::kLaunch);
  return e;
}

template <int TY, int S, int MINB>
static cudaError_t launch_t(const PropLaunch &L, cudaStream_t s) {
  constexpr size_t smem = smem_bytes<TY, S>();
  static bool ready = false;  // dynamic shared-memory limit set for this shape
  if (!ready) {
    cudaError_t e = prepare_t<TY, S, MINB>();
    if (e != cudaSuccess) return e;
    ready = true;
  }
  const bool iso = L.p.iso != 0;
  auto kern = L.batch ? (iso ? k_propagate_fp32<TY, S, true, true, MINB> : k_propagate_fp32<TY, S, false, true, MINB>)
                      : (iso ? k_propagate_fp32<TY, S, true, false, MINB> : k_propagate_fp32<TY, S, false, false, MINB>);
  return launch_step(kern, L.grid, propagate_fp32_threads(TY), smem, s, L.m, L.p);
}

// Supported shapes: rows per tile x stages.  Tiles of 16 and 12 rows run one
// CTA per SM, tiles of 8 rows two.
#define FLT_SHAPES(X) X(12, 4, 1) X(12, 5, 1) X(12, 6, 1) X(16, 4, 1) X(16, 5, 1) X(8, 4, 2) X(8, 5, 2)

size_t propagate_fp32_smem_bytes(int ty, int st) {
#define X(a, b, c) \
  if (ty == a && st == b) return smem_bytes<a, b>();
  FLT_SHAPES(X)
#undef X
  return 0;
}
bool propagate_fp32_supported(int ty, int st) { return propagate_fp32_smem_bytes(ty, st) != 0; }
int propagate_fp32_threads(int ty) { return kTileX * ((ty / 2 + 3) / 4 * 4 + kHelperWarps); }
int propagate_fp32_ctas_per_sm(int ty) { return ty == 8 ? 2 : 1; }

cudaError_t propagate_fp32_prepare(int ty, int st) {
#define X(a, b, c) \
  if (ty == a && st == b) return prepare_t<a, b, c>();
  FLT_SHAPES(X)
#undef X
  return cudaErrorInvalidValue;
}

// The fault-injection variant: the default shape, single shot.
static cudaError_t launch_hook(const PropLaunch &L, cudaStream_t s) {
  constexpr int TY = 16, S = 5;
  constexpr size_t smem = smem_bytes<TY, S>();
  // Any pipeline depth of the step's own shape: the plan depends on the rows
  // only.  (The coefficient planes are present in either layout.)
  if (L.batch || L.tile_rows != TY) return cudaErrorInvalidValue;
  auto kern = L.p.iso ? k_propagate_fp32<TY, S, true, false, 1, true> : k_propagate_fp32<TY, S, false, false, 1, true>;
  const cudaError_t e = prepare_step_kernel((const void *)kern, smem, Regs<TY>::kLaunch);
  if (e != cudaSuccess) return e;
  return launch_step(kern, L.grid, propagate_fp32_threads(TY), smem, s, L.m, L.p);
}

// The media-table layout: single shot, 16-row tiles.
#define FLT_MEDIA_SHAPES(X) X(16, 5) X(16, 6) X(16, 7)

template <int TY, int S>
static cudaError_t launch_media_t(const PropLaunch &L, cudaStream_t s) {
  constexpr size_t smem = smem_bytes<TY, S, true>();
  static_assert(smem <= 227 * 1024, "media-table shape exceeds the shared memory of a CTA");
  auto kern_i = k_propagate_fp32<TY, S, true, false, 1, false, true>;
  auto kern_a = k_propagate_fp32<TY, S, false, false, 1, false, true>;
  static bool ready = false;
  if (!ready) {
    for (auto kern : {kern_i, kern_a}) {
      const cudaError_t e = prepare_step_kernel((const void *)kern, smem, Regs<TY>::kLaunch);
      if (e != cudaSuccess) return e;
    }
    ready = true;
  }
  return launch_step(L.p.iso ? kern_i : kern_a, L.grid, propagate_fp32_threads(TY), smem, s, L.m, L.p);
}

bool propagate_fp32_media_supported(int ty, int st) {
#define X(a, b) \
  if (ty == a && st == b) return true;
  FLT_MEDIA_SHAPES(X)
#undef X
  return false;
}

cudaError_t propagate_fp32_launch(const PropLaunch &L, cudaStream_t s) {
  if (L.d1d1) return propagate_d1d1_launch(L, s);
  if (fault_injected(L.p)) return launch_hook(L, s);
  if (L.media) {
    if (L.batch || !L.p.media) return cudaErrorInvalidValue;
#define X(a, b) \
  if (L.tile_rows == a && L.stages == b) return launch_media_t<a, b>(L, s);
    FLT_MEDIA_SHAPES(X)
#undef X
    return cudaErrorInvalidValue;
  }
#define X(a, b, c) \
  if (L.tile_rows == a && L.stages == b) return launch_t<a, b, c>(L, s);
  FLT_SHAPES(X)
#undef X
  return cudaErrorInvalidValue;
}

}  // namespace flt
