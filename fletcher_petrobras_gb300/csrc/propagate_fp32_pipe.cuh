// Pipeline pieces of the FP32 step kernels (propagate_fp32.cu,
// propagate_d1d1.cu): the shared-memory stage layout, the work items of a
// launch, and the producer's TMA issue of one step.
#pragma once
#include "device_util.cuh"
#include "fletcher_internal.h"

namespace flt {

// Plane k arrives at step k; plane k - kLag is updated at that step.  Its
// z stencil (planes k-kLag-4 .. k-kLag+4) lives in per-thread rings of
// kRing planes, and its in-plane terms in kABSlots shared-memory slots.
constexpr int kLag = 4;
constexpr int kRing = kLag + 5;
constexpr int kABSlots = kLag + 1;

template <int TY, bool D1D1 = false, bool MT = false>
struct Geo {
  static constexpr int TX = kTileX;
  static constexpr int HX = TX + 2 * kRadius;
  static constexpr int HY = TY + 2 * kRadius;
  static constexpr int NT = TX * TY;
  static constexpr int HALO_B = HX * HY * 8;
  static constexpr int ARR_B = MT ? 0 : kArrivalCoef * NT * 4;
  static constexpr int UPD_B = (MT ? kVelCoef : kUpdateCoef) * NT * 4;  // media table: velocity terms only
  static constexpr int PP_B = NT * 8;
  static constexpr int ID_B = MT ? NT : 0;  // medium ids, one byte per cell
  static constexpr int OFF_ARR = HALO_B;
  static constexpr int OFF_UPD = OFF_ARR + ARR_B;
  static constexpr int OFF_PP = OFF_UPD + UPD_B;
  static constexpr int OFF_IDC = OFF_PP + PP_B;  // ids of plane k
  static constexpr int OFF_IDU = OFF_IDC + ID_B;  // ids of plane k-4
  static constexpr int STAGE_B = (OFF_IDU + ID_B + 127) / 128 * 128;
  static constexpr int TAB_B = MT ? kAngleCoef * kMediaMax * 4 : 0;
  // One exchange buffer: D1y of the tile rows with their 4-column x halo, or
  // (Der1-Der1 numerics) D1x of the tile columns with their 4-row y halo.
  static constexpr int ROW_B = D1D1 ? HY * TX * 8 : TY * HX * 8;
  static_assert(TY % 4 == 0, "tile rows must be a multiple of 4");
  static_assert(HALO_B % 128 == 0 && ARR_B % 128 == 0 && UPD_B % 128 == 0 && ID_B % 128 == 0,
                "stage regions 128-B aligned");
  static_assert(!(MT && D1D1), "the Der1-Der1 numerics read the coefficient planes");
};

// A work item: a z range [z0, z1) of the tile column at (x0, y0) of a shot,
// stored as a segment {x0, y0, z0, z1}, in batched launches {tile x index +
// (shot << 16), y0, z0, z1}.  CTA b of a launch takes the segments
// P.cta_first[b] .. P.cta_first[b + 1] - 1 of P.seg.
struct Item {
  int x0, y0, z0, z1;
  int shot;
};

template <bool BATCH>
__device__ __forceinline__ Item decode_item(int4 w) {
  Item it;
  it.x0 = BATCH ? kRadius + (w.x & 0xffff) * kTileX : w.x;
  it.y0 = w.y;
  it.z0 = w.z;
  it.z1 = w.w;
  it.shot = BATCH ? int((unsigned)w.x >> 16) : 0;
  return it;
}

// Descriptors used for one step of item `it` (ids, vel: media-table layout).
struct StepMaps {
  const CUtensorMap *cur, *prev, *arr, *upd, *ids, *vel;
};

// Issues the TMA loads of one step (plane k of item `it`) into `stage`.
// Media-table layout: the id tiles start at column x0 + kIdShift of the id
// volume (x0 = kRadius + 32 t, so a multiple of 16 bytes).
template <int TY, bool MT = false>
__device__ __forceinline__ void issue_step(unsigned char *stage, uint64_t *bar, const Item &it, int k,
                                           const StepMaps &m) {
  using G = Geo<TY, false, MT>;
  const bool center = (k >= it.z0) && (k < it.z1);
  const bool upd = (k - kLag >= it.z0);
  const uint32_t bytes =
      G::HALO_B + (center ? G::ARR_B + G::ID_B : 0) + (upd ? G::UPD_B + G::PP_B + G::ID_B : 0);
  const int ct = (it.x0 - kRadius) / kTileX;  // tile column in the coefficient block
  mbar_arrive_expect_tx(bar, bytes);
  tma_load_3d(stage, m.cur, bar, it.x0 - kRadius, it.y0 - kRadius, k);
  if constexpr (MT) {
    if (center) tma_load_3d(stage + G::OFF_IDC, m.ids, bar, it.x0 + kIdShift, it.y0, k);
    if (upd) {
      tma_load_4d(stage + G::OFF_UPD, m.vel, bar, DC_V2PX * kTileX, ct, it.y0, k - kLag);
      tma_load_3d(stage + G::OFF_IDU, m.ids, bar, it.x0 + kIdShift, it.y0, k - kLag);
      tma_load_3d(stage + G::OFF_PP, m.prev, bar, it.x0, it.y0, k - kLag);
    }
  } else {
    if (center) tma_load_4d(stage + G::OFF_ARR, m.arr, bar, 0, ct, it.y0, k);
    if (upd) {
      tma_load_4d(stage + G::OFF_UPD, m.upd, bar, kArrivalCoef * kTileX, ct, it.y0, k - kLag);
      tma_load_3d(stage + G::OFF_PP, m.prev, bar, it.x0, it.y0, k - kLag);
    }
  }
}

}  // namespace flt
