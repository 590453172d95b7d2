// Internal interfaces between the C-ABI layer (driver.cu) and the kernels.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace flt {

constexpr int kRadius = 4;   // stencil half-width of Der2 / DerCross
constexpr int kTileX = 32;   // tile width in x: one warp per tile row
constexpr int kNumCoef = 10;

// Device coefficient block layout: [z][y][t][c][32], c in this order and t the
// tile column of the step kernels (32 cells, from x = kRadius + 32 t; the
// kRadius columns before the first tile, which no step reads, follow the row's
// last cell), so that the coefficients a tile row needs together are
// contiguous: 384 bytes of the first three, read when a plane arrives (in-plane
// terms), and 896 of the other seven, read when the plane is updated four planes
// later.  Against ten separate planes ([z][c][y][x], 128 bytes at a time), of
// the same size: 504^3 1.865 -> 1.792 ms a step (and up to 2.03 ms before on
// other boxes), 128^3 + shell 82.0 -> 76.4 us.
enum DevCoef {
  DC_XX = 0, DC_YY, DC_XY,                    // arrival: ch1dxx ch1dyy ch1dxy
  DC_ZZ, DC_XZ, DC_YZ, DC_V2PX, DC_V2PZ, DC_V2SZ, DC_V2PN  // update
};
__host__ __device__ inline int coef_tiles(int pitch) { return pitch / kTileX; }
// Floats of the block; column of cell x in its row; index of coefficient 0 of a
// column of row (y, z), that of coefficient c being kTileX * c further.
__host__ __device__ inline size_t coef_floats(int sy, int sz, int pitch) {
  return (size_t)sz * sy * coef_tiles(pitch) * (kNumCoef * kTileX);
}
__host__ __device__ inline int coef_column(int x, int sx) { return x >= kRadius ? x - kRadius : sx - kRadius + x; }
__host__ __device__ inline size_t coef_index(int xs, int y, int z, int sy, int pitch) {
  return (((size_t)z * sy + y) * coef_tiles(pitch) + xs / kTileX) * (kNumCoef * kTileX) + xs % kTileX;
}
constexpr int kArrivalCoef = 3;
constexpr int kUpdateCoef = 7;

// Media-table layout of the coefficients (FP32 form): the six angle terms
// (DC_XX .. DC_YZ) depend on a cell's (phi, theta) only, so a model with at
// most kMediaMax distinct (phi, theta) pairs stores them once per pair in a
// table [6][kMediaMax] and one byte per cell (the pair's slot) in an id
// volume [z][y][ipitch].  The id of cell x sits in byte x + kIdShift of its
// row: a tile's first column kRadius + 32 t then starts at a multiple of 16
// bytes, as a TMA load of 8-bit elements needs.  The four velocity terms
// (DC_V2PX .. DC_V2PN) stay per cell in the coefficient block.
constexpr int kMediaMax = 256;
constexpr int kAngleCoef = 6;
constexpr int kVelCoef = 4;
constexpr int kIdShift = 12;
// Default pipeline depth of the media-table layout.  5, 6 and 7 stages, us a
// step: 504^3 1487, 1573 and 1571, 272^3 updated cells 176, 193 and 189, 192^3
// 63.7, 63.1 and 63.5 (with more stages the CTAs run further apart and share
// less in L2).
constexpr int kMediaStages = 5;
static_assert((kRadius + kIdShift) % 16 == 0 && kTileX % 16 == 0, "id tiles must start on 16-byte boundaries");
static_assert(DC_V2PX == kAngleCoef && DC_V2PN == kNumCoef - 1, "velocity terms follow the angle terms");

// One shot's geometry and buffers, in device memory (read by every launch).
// The fields are stored as (p, q) pairs of float, [z][y][pitch] with x fastest.
struct ShotDesc {
  float2 *F[2];                  // the two field buffers
  int sx, sy, sz, pitch, bord;
  int src_x, src_y, src_z;       // cell that gains the step's source (src_z < 0: none)
  int cor_x, cor_y, cor_z;       // cell whose previous-field value lacks the last step's
                                 //   source (added on read; cor_z < 0: none)
  int pad[2];
};

// TMA descriptors of one shot (in device memory; CUtensorMap carries the
// alignment TMA needs).
struct ShotMaps {
  CUtensorMap halo[2];  // field buffer b, box (TX+8, TY+8, 1)
  CUtensorMap pt[2];    // field buffer b, box (TX, TY, 1)
  CUtensorMap arr;      // coefficients, box (TX * 3, 1, TY, 1) of (coefficients, tile, y, z)
  CUtensorMap upd;      // coefficients, box (TX * 7, 1, TY, 1)
};

// One launch: every active shot advances one step.  The work is a list of
// segments, each a z range of one tile column of a shot: {x0, y0, z0, z1}, in
// batched launches {tile x index + (shot << 16), y0, z0, z1}.  CTA b takes
// the segments cta_first[b] .. cta_first[b+1]-1.
struct PropParams {
  ShotDesc one;                     // single-shot launches: the shot itself
  const ShotDesc *shots;            // batched launches: per-shot descriptors
  const ShotMaps *maps;
  int parity;                       // current field = F[parity], previous = F[1 - parity]
  float inv_dx, inv_dy, inv_dz;     // 1/dx, 1/dy, 1/dz
  float inv_dxx, inv_dyy, inv_dzz;  // 1/(dx*dx), 1/(dy*dy), 1/(dz*dz) as the reference forms them
  float inv_dxy, inv_dxz, inv_dyz;  // 1/(dx*dy), 1/(dx*dz), 1/(dy*dz): factors of the cross derivatives
  int iso;                          // dx == dy == dz: derivatives unscaled, dt2 = dt^2 / h^2
  float dt2;                        // factor of the rhs in the update
  float dt;                         // the time step (Der1-Der1 numerics: rhs * dt * dt)
  float src;                        // value added at each shot's source cell (src_z >= 0)
  float cor;                        // value owed at each shot's cor cell (cor_z >= 0)
  unsigned int *err;                // error word (bit 0: bounded wait gave up)
  const int4 *seg;                  // the segment list
  const int *cta_first;             // its [grid + 1] first segments
  int skip_rows;                    // warps whose row lies outside the updated region do not compute
  const float *media;               // media-table layout: angle terms [kAngleCoef][kMediaMax]
  // Fault injection (tests; -1: none): CTA 0 skips the loads of its
  // stall_step-th step; one of its helper warps gives up at its quit_step-th;
  // the launch's waits are limited to wait_tries tries (mbar_spin).
  int stall_step, quit_step;
  unsigned wait_tries;
};

// The four descriptors a single-shot launch passes as kernel parameters.
struct SingleMaps {
  CUtensorMap cur_halo, prev_pt, arr, upd;
  CUtensorMap ids, vel;  // media-table layout: id volume, box (TX, TY, 1); velocity terms, box (TX * 4, 1, TY, 1)
};

struct PropLaunch {
  PropParams p;
  SingleMaps m;           // single-shot launches
  bool batch;             // true: p.shots / p.maps describe the shots
  bool d1d1;              // Der1-Der1 numerics (single shot, 16 x 4 tiles)
  bool media;             // media-table coefficient layout (single shot)
  int tile_rows;          // TY
  int stages;
  int grid;
};

// Launches a step kernel so that its CTAs may start, and set themselves up
// (barriers, tensor maps, work lists), as CTAs of the launch before it in
// the stream leave; the kernel waits for that launch to complete before it
// touches fields, scales or maxima.  Saves about 2 us of every step: 56^3 +
// shell 14.4 -> 12.5 us, 128^3 + shell 76.4 -> 73.6, 272^3 updated cells 207
// -> 205; at 504^3 nothing (1.79 ms).
template <class... K, class... A>
inline cudaError_t launch_step(void (*kern)(K...), int grid, int block, size_t smem, cudaStream_t s, const A &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

// Before a step kernel's first launch: its dynamic shared-memory limit, and a
// check of its register split.  setmaxnreg moves registers between the warps of
// a CTA within what the launch gives them; a kernel compiled to fewer than
// `launch_regs` a thread would leave setmaxnreg.inc waiting without limit.
inline cudaError_t prepare_step_kernel(const void *kern, size_t smem, int launch_regs) {
  cudaFuncAttributes a;
  const cudaError_t e = cudaFuncGetAttributes(&a, kern);
  if (e != cudaSuccess) return e;
  if (a.numRegs < launch_regs) return cudaErrorInvalidKernelImage;
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

inline bool fault_injected(const PropParams &P) { return P.stall_step >= 0 || P.quit_step >= 0; }

size_t propagate_fp32_smem_bytes(int tile_rows, int stages);
bool propagate_fp32_supported(int tile_rows, int stages);
// Shapes built for the media-table layout.
bool propagate_fp32_media_supported(int tile_rows, int stages);
int propagate_fp32_threads(int tile_rows);
int propagate_fp32_ctas_per_sm(int tile_rows);
cudaError_t propagate_fp32_prepare(int tile_rows, int stages);
cudaError_t propagate_fp32_launch(const PropLaunch &L, cudaStream_t s);
cudaError_t propagate_d1d1_launch(const PropLaunch &L, cudaStream_t s);
// Working sets below this stay in the 129 MB L2 from step to step.
constexpr double kL2Bytes = 100e6;
// Tile shape of the Der1-Der1 numerics (the only one built for it).
constexpr int kD1D1Rows = 16, kD1D1Stages = 4;
// Most concurrent chains of the batched shots' chain schedule, and the
// updated cells from which a shot fills the GPU on its own and up to which
// two chains beat one.  Persistent launch / one chain / two chains, us a step:
// 12 shots of 1.2 M cells 199 / 218 / 209, 8 of 2.4 M 245 / 256 / 246, 3 of
// 4.4 M 159 / 162 / 159, 4 of 6.6 M 296 / 302 / 291, 5 of 10 M 562 / 566 / 548,
// 6 of 17 M 1083 / 1083 / 1080, 2 of 26 M 551 / 551 / 564, 3 of 26 M 828 / 826 /
// 839; FP16 2 of 17 M 402 / 402 / 386, 3 of 26 M 912 / 898 / 887.
constexpr int kMaxChains = 8;
constexpr double kChainFillCells = 2.1e6, kTwoChainCells = 20e6;

// ---- 16-bit field storage (propagate_half.cu) ----
// A field buffer holds (p, q) as half2 per cell ([z][y][pitch]) and, in the
// extended form, one residual byte per value (a ushort per cell), with a
// power-of-two scale per z-plane.
struct HalfMaps {
  CUtensorMap cur_hi, cur_lo;    // current field, halo box (TX+8, TY+8, 1)
  CUtensorMap prev_hi, prev_lo;  // previous field: box (TX, TY, 1) / residuals (TX+8, TY, 1) from x0-4
  CUtensorMap arr, upd;          // coefficients, as in the FP32 form
};

// One batched shot of a 16-bit form (device memory).
struct HalfShot {
  unsigned *hi[2];        // the two field buffers: (p, q) as half2 per cell
  unsigned short *lo[2];  // their residual bytes (extended form; null otherwise)
  int *E;                 // [3][sz] per-plane exponents; the field of step it uses slot it % 3
  unsigned *Mx;           // per-plane max |value| (float bits): persistent steps [2][sz], of the field in
                          //   buffer b; chained steps [4][sz], of the field of step it in slot it % 4
};

// A batched shot's tensor maps, by the buffer that holds the current field.
struct HalfShotMaps {
  HalfMaps m[2];
};

struct HalfParams {
  PropParams p;                       // geometry (p.one), spacing, source, error word
  unsigned *out_hi;                   // new field: half2 per cell
  unsigned short *out_lo;             // new field: residual bytes (extended form)
  const int *e_cur, *e_prev;          // per-plane exponents of the current and previous field
  int *e_new;                         // those of the new field (FP16X: set by the step itself)
  // Per-plane max |value| (float bits) of the current and previous field, of
  // the new one (atomicMax, cleared by the step before), and the slot this
  // step clears for the next.
  const unsigned *m_cur, *m_prev;
  unsigned *m_new, *m_clear;
  // Batched launches (p.shots): per-shot buffers and maps, and the
  // exponent slot of the current field (step % 3).
  const HalfShot *hshots;
  const HalfShotMaps *hmaps;
  int ecur;
};

struct HalfLaunch {
  HalfParams h;
  HalfMaps m;
  int tile_rows, stages, grid;
  bool batch;  // h.p.shots / h.hshots / h.hmaps describe the shots
};

bool propagate_half_supported(int tile_rows, int stages);
// One 16-bit step; FP16 single shots: preceded by the launch that sets the new
// planes' exponents (in batches half_scales_batch does).
cudaError_t propagate_half_launch(const HalfLaunch &L, bool ext, cudaStream_t s);
cudaError_t propagate_half_prepare(int tile_rows, int stages, bool ext, bool batch);
// Before a batched 16-bit step: the new field's plane exponents and the
// cleared maxima of the first `active` shots of `order`,
// block i taking shot order[i]; the current field is in buffer c, its
// exponents in slot ecur.
cudaError_t half_scales_batch(const HalfShot *hs, const ShotDesc *sd, const int *order, int active, int c, int ecur,
                              float src_abs, cudaStream_t s);
cudaError_t half_encode(const float *p, const float *q, unsigned *hv, unsigned short *rv, int *e, unsigned *m, int sx,
                        int sy, int sz, int pitch, bool ext, cudaStream_t s);
cudaError_t half_decode(const unsigned *hv, const unsigned short *rv, const int *e, float *out, int comp, int sx,
                        int sy, int sz, int pitch, bool ext, int grid, cudaStream_t s);

// ---- learned absorbing boundary (abc_learned.cu) ----
// The resident single-shot state as the boundary layer sees it.
struct ResidentView {
  bool init = false;
  int sx = 0, sy = 0, sz = 0, bord = 0, pitch = 0;
  float dx = 0, dy = 0, dz = 0, dt = 0;
  const float2 *cur = nullptr, *prev = nullptr;  // current and previous (p, q) fields (FP32 form)
  float2 *next = nullptr;                        // the buffer the step writes
  const float *coef = nullptr;                   // coefficient block (DevCoef order)
  cudaStream_t stream = nullptr;
  int num_sms = 0;
  unsigned *err = nullptr;                       // the error word (bit 0: a bounded wait gave up)
};
ResidentView resident_view();       // driver.cu; cur/prev/next for the next step
bool abc_active();                  // a boundary layer is set on the resident state
cudaError_t abc_after_step(const ResidentView &v);   // the layer's update of next, after the plain step
void abc_release_resident();        // the resident state is re-initialised or finalised

// ---- output path (snapshot.cu) ----
// Field `which` (0 current p, 1 current q, 2 previous p, 3 previous q) of the
// resident state, any storage form, as an unpitched FP32 volume in dev_out,
// issued on the library's stream.  fix_idx / fix_val: the one cell whose
// stored value lacks a source addition the interface shows (-1: none).
int resident_field_to_device(int which, float *dev_out, long *fix_idx, float *fix_val);
size_t resident_cells();             // sx * sy * sz (0 when not initialised)
bool resident_dims(int *sx, int *sy, int *sz);  // grid of the resident state (any form)
cudaStream_t resident_stream();      // the library's stream
void snapshot_release();             // driver.cu calls it when the state goes away

// Time limit of the learned layer's grid barriers (ns); the step kernels count
// their tries instead (mbar_spin).
constexpr uint64_t kWaitLimitNs = 2000000000ull;
// Limit of an aborting producer's wait for each stage's loads (ns).
constexpr uint64_t kDrainNs = 200000000ull;

}  // namespace flt
