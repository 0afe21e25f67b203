// Host-side state of one scene handle and the per-storage-type kernel
// launcher interface.  Shared by the C ABI (lbm_capi.cu) and the typed
// launchers (lbm_inst_*.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "lbm_b200.h"
#include "lbm_core.cuh"

struct lbm_sim;

namespace lbm {

// Launch configuration of the fused step kernel.
struct FusedCfg {
  int ty = 4;       // tile shape: cell rows per CTA (CTA = 32 x (rows + 2) threads),
                    // | LBM_FUSED_COMPACT / _ASYNC / _STAGED / _TMA for the compact-ring forms
  int zchunk = 32;  // z planes marched per CTA
  bool set = false; // by the caller (else auto_zchunk's)
};

// z planes per CTA for a launch of tiles(z) CTAs, each of which collides two
// planes more than it writes, on `sms` SMs of which each holds `perSM` CTAs.
// The cost of a choice is its planes per CTA times the waves of CTAs, in the
// time a plane takes on a full SM:
//   * one CTA on an SM takes 0.65 of that a plane (measured 2.1 us alone
//     against 3.2 us for two, 6 compact rows);
//   * up to two waves the last wave counts whole;
//   * of more waves it counts a quarter of what it is short, since the CTAs
//     are no longer in step by then;
//   * from eight waves on only the two extra planes are left, and chunks
//     longer than zmany read apart from their neighbours: zmany (22 planes
//     FP32, 24 FP16 at 256^3, 14 waves, the best of 16 to 32).
// Measured step without spheres, before (z-chunks of 22 / 24) and with the
// rule: 40x28x40 44.7 -> 13.3 us (3 planes), 61x47x83 51.0 -> 23.8 (5),
// 80x72x96 66.9 -> 48.7 (12), 128x97x110 FP16 110.0 -> 98.9 (27), 160x112x160
// 201.2 -> 191.4 (27); against the best of every length the rule is within 9%
// from 12^3 to 192x160x176.
template <class Tiles>
inline int auto_zchunk(int planes, int zmany, int perSM, int sms, Tiles &&tiles) {
  constexpr int ZMAX = 32;
  const double slots = (double)perSM * sms, alone = perSM > 1 ? 0.65 : 1.0;
  if (tiles(zmany) >= 8 * slots) return zmany;
  int best = 1;
  double least = 0;
  for (int z = 1; z <= planes && z <= ZMAX; z++) {
    const double n = (double)tiles(z), w = n / slots, f = w - (long long)w;
    double eff;
    if (n <= sms) eff = alone;
    else if (w <= 1) eff = 1;
    else if (w < 2) eff = 1 + (f <= 0.5 ? alone : 1);
    else eff = f > 0 ? w + 0.25 * (1 - f) : w;
    const double cost = (z + 2) * eff;
    if (z == 1 || cost <= least) best = z, least = cost;
  }
  return best;
}
// equal chunks of at most zmax planes
inline int even_zchunk(int planes, int zmax) {
  const int chunks = (planes + zmax - 1) / zmax;
  return chunks > 0 ? (planes + chunks - 1) / chunks : 1;
}

// cell rows per CTA of a tile shape
inline int shape_rows(int shape) { return shape & 0xff; }
// internal shape bit: the launch covers a grid whose D3Q27 populations exceed
// 2^31 elements, so the fused kernel uses 64-bit population offsets
constexpr int SHAPE_WIDE = 0x200;
inline bool needs_wide(long long cells) { return pop_elems(cells, 27) >= (1LL << 31) - 64; }


// A step's shell launch (lbm_shell.cuh): the step's spheres, the 1,024-cell
// chunks of the largest one's box, and in the device-resident loop (tail) the
// sphere step and the next plan, with slotCells impulse slots per sphere and
// retag boxes of at most maxU cells.
struct StepCtx {
  int ns = 0, redChunks = 0;
  bool tail = false;
  bool anyTag = false;  // the tags may not be the plan's
  long long slotCells = 0, maxU = 0;
};

class OpsBase {
 public:
  virtual ~OpsBase() {}
  virtual size_t pop_bytes() const = 0;    // bytes per stored population
  virtual size_t macro_bytes() const = 0;  // bytes per macro value
  virtual bool phases_supported() const = 0;
  virtual void init_flat(lbm_sim *h, const double *d_phiCol) = 0;
  virtual void seed_hydrostatic(lbm_sim *h) = 0;
  virtual void gradients(lbm_sim *h) = 0;
  // Kernels of a step read the sphere set and boxes from h->dPlan.
  virtual void retag_full(lbm_sim *h) = 0;
  // retag from a host-evaluated solid mask and surface velocities (device copies)
  virtual void retag_mask(lbm_sim *h, const uint8_t *d_mask, const float *d_us) = 0;
  // momentum-exchange links of the last phase-by-phase hydro stream, scan order
  virtual void link_count(lbm_sim *h, int *d_chunks) = 0;
  virtual void link_emit(lbm_sim *h, const int *d_chunks, int cap, int *cells, int8_t *dirs, double *mom) = 0;
  virtual void collide_phase(lbm_sim *h) = 0;
  virtual void stream_phase(lbm_sim *h) = 0;
  virtual void collide_hydro(lbm_sim *h) = 0;
  virtual void stream_hydro_macro(lbm_sim *h) = 0;
  // the cells of [c0, c1) that a step does not update: current half -> the other
  virtual void carry_solid(lbm_sim *h, long long c0, long long c1) = 0;
  // retag on the plan's box (retag), fresh / dead lists, fresh fill (fill)
  virtual void sets(lbm_sim *h, long long maxChunks, bool retag, bool fill) = 0;
  virtual void absorb_dead(lbm_sim *h, double *d_out) = 0;
  virtual void fused_step(lbm_sim *h, const FusedCfg &cfg) = 0;
  virtual void shell(lbm_sim *h, const StepCtx &c) = 0;  // after fused_step, before cur flips
  virtual void finish_unowned(lbm_sim *h) = 0;           // after shell, where the tags may not be the plan's
  virtual void pack(lbm_sim *h, uint8_t *d_out) = 0;
  virtual void pack_end_planes(lbm_sim *h, uint8_t *d_out) = 0;
  virtual void watch_finite(lbm_sim *h, unsigned long long *d_first) = 0;
  // Reference-layout float32 <-> device storage for population fields.
  // half: 0 = both halves (current state), 1 = [cur], 2 = [1-cur].
  virtual void upload_pops(lbm_sim *h, bool isH, int half, const float *d_aos, long long c0,
                           long long cells) = 0;
  virtual void download_pops(lbm_sim *h, bool isH, int half, float *d_aos, long long c0,
                             long long cells) = 0;
  virtual void download_pops64(lbm_sim *h, bool isH, int half, double *d_aos, long long c0,
                               long long cells) = 0;
  // Re-express h offsets after phi changed from d_oldPhi (both halves).
  virtual void reencode_h(lbm_sim *h, int half, const void *d_oldPhi) = 0;
  // Fused-step kernel geometry (for the bench and the autotuner).
  virtual size_t fused_smem(int ty) const = 0;
  // Batched fused step: per-scene descriptors (FusedArgs of this storage type,
  // fused_args_bytes() each) for a given ping-pong half, and one persistent
  // launch over the tiles of every scene.
  virtual size_t fused_args_bytes() const = 0;
  virtual void fused_args(lbm_sim *h, int cur, int zchunk, void *out) = 0;
  virtual int fused_batch_ctas(int ty, int device) = 0;  // resident CTAs on the device
  virtual void fused_batch(const void *d_args, const int *d_tileStart, const int3 *d_tileGrid,
                           int nscenes, int ty, int ctas, cudaStream_t st) = 0;
  // Fault record of the bounds-checked build (all zero otherwise); cleared on read.
  virtual cudaError_t read_fault(lbm_sim *h, unsigned long long out[4]) = 0;
  // a tile shape this storage form supports (rows 2, 4, 8; 4 | LBM_FUSED_STAGED for FP16/BF16)
  virtual bool shape_ok(int shape) const = 0;
  // load every fused step and batch kernel instance of this storage form on
  // the device (and set their shared-memory opt-in), so that no first launch
  // waits for a module load
  virtual void warm(int device) = 0;
  // ux and uy held in the population pad slots (FP32 / FP64 storage), and
  // their copy to or from a plain array of one half (the field transfers)
  virtual bool u_in_pads() const = 0;
  virtual void u_array(lbm_sim *h, int comp, int half, void *arr, bool toScene) = 0;
  // a batch's sparse work, one launch per kind for all scenes: the per-scene
  // argument blocks, the first plans, then per step the retag, fresh / dead
  // sets and fresh fill before the fused launch and the shells after it
  virtual size_t small_args_bytes() const = 0;
  virtual size_t shell_args_bytes() const = 0;
  virtual void small_args(lbm_sim *h, int cur, void *out) = 0;
  virtual void shell_args(lbm_sim *h, const StepCtx &c, int cur, void *out) = 0;
  virtual void batch_plan(const void *d_shell, int n, cudaStream_t st) = 0;
  // (inOrder: a scene has the test hook's fill)
  virtual void batch_sets(const void *d_small, int n, unsigned ctas, bool inOrder, cudaStream_t st) = 0;
  virtual void batch_shell(const void *d_shell, int n, int redChunks, int spheres, cudaStream_t st) = 0;
  // the tensor maps of the TMA-staged form (h->dMaps), where the storage
  // form and the grid allow them (nx a multiple of 16); none otherwise
  virtual int build_stage_maps(lbm_sim *) { return 0; }
};

OpsBase *make_ops_f32();
OpsBase *make_ops_f16();
OpsBase *make_ops_bf16();
OpsBase *make_ops_f64();

}  // namespace lbm

struct lbm_sim {
  int nx = 0, ny = 0, nz = 0, storage = 0, device = 0;
  long long n = 0;
  cudaStream_t stream = nullptr;
  lbm_params params{};
  int cur = 0;
  lbm::OpsBase *ops = nullptr;
  lbm::FusedCfg cfg;
  bool fusedOK = true;  // the fused kernel's 32-bit indexing covers this grid
  bool withholdStage = false;  // test hook: the staged fused kernel withholds its first copy

  // device memory
  void *F[2] = {nullptr, nullptr};
  void *H[2] = {nullptr, nullptr};
  void *mac[2][5] = {{nullptr}};  // phi, rho, ux, uy, uz
  uint8_t *tag = nullptr, *tagPrev = nullptr;
  void *grad[4] = {nullptr};  // gx gy gz lap (phase-by-phase scratch)
  void *us[3] = {nullptr};
  void *bf[3] = {nullptr};
  bool bfActive = false;

  int *fresh = nullptr, *dead = nullptr;  // scan-ordered lists
  long long listCap = 0;
  int2 *counts = nullptr;  // per compaction chunk
  void *setBits = nullptr; // per compaction chunk: its fresh / dead ballot words
  long long countsCap = 0;
  int *totals = nullptr;  // device [3]: n_fresh, n_dead, fused-step status (non-zero: a bounded wait ran out)
  bool listsValid = false;

  double *impAcc = nullptr;  // per-cell impulse slots of every sphere
  long long impCap = 0;      // doubles
  double *partials = nullptr;
  void *dMaps = nullptr;    // tensor maps of the TMA-staged form (device memory), or null
  void *meshTri = nullptr;  // a mesh's triangles for lbm_voxelize_mesh / lbm_retag_cells_mesh
  size_t meshCap = 0;
  unsigned *redTickets = nullptr;  // last-block tickets: [LBM_MAX_SPHERES] of the impulse sums, one of the sets kernel
  long long partialsCap = 0;  // doubles
  int partialsChunks = 0;
  double *dOut = nullptr;      // device [2][MAX][6]: fluid impulses, dead impulses
  double *hOut = nullptr;      // pinned host mirror
  lbm_sphere *dSph = nullptr;  // device sphere array for the coupled loop
  lbm::Plan hPlan{};           // host copy of the step plan
  lbm::Plan *dPlan = nullptr;  // [2] device step plans: the step that reads half c uses plan c
  lbm::Plan *plan() const { return dPlan + cur; }
  void *staging = nullptr;
  size_t stagingBytes = 0;
  void *image = nullptr;  // rendered RGBA8 frame (lbm_render)
  // lbm_pack_volume_async / lbm_step_frame: packed frames on the device, two
  // used in turn, each copied to the host on copyStream; evPacked orders a
  // copy after its pack, evFrame[b] the next pack into buffer b after b's
  // copy, evCopied marks the last copy issued
  void *frameDev[2] = {nullptr, nullptr};
  cudaEvent_t evFrame[2] = {nullptr, nullptr};
  cudaEvent_t evPackedSlot[2] = {nullptr, nullptr};
  bool framePending[2] = {false, false};
  int frameNext = 0;
  // lbm_step_frame's copy to the host, issued when the next step's fused
  // kernel is queued (so it runs beside that kernel, not ahead of the step's
  // small read-backs on the same copy engine); -1: none waiting
  int deferredSlot = -1;
  uint8_t *deferredHost = nullptr;
  cudaStream_t copyStream = nullptr;
  cudaEvent_t evPacked = nullptr, evCopied = nullptr;
  bool copyPending = false;
  size_t imageBytes = 0;
  double *dPhiCol = nullptr;
  int *hTotals = nullptr;  // pinned [3]
  // NaN/Inf watchdog (lbm_set_nan_watchdog): off while watchEvery is 0
  int watchEvery = 0;
  long long watchSteps = 0;            // steps completed since the last scan
  unsigned long long *dWatch = nullptr;  // device: lowest non-finite cell index

  lbm::Box boxLast{{1, 1, 1}, {0, 0, 0}};
  lbm::Box boxLastLast{{1, 1, 1}, {0, 0, 0}};
  lbm::Box lastRetagBox{{1, 1, 1}, {0, 0, 0}};
  // a step split by lbm_step_begin / lbm_step_end: the spheres' box of the
  // begun step, and how many spheres it was begun with (-1: none begun)
  lbm::Box stepNow{{1, 1, 1}, {0, 0, 0}};
  // a frame step: the fused kernel writes the step's RG8 volume here
  // (planes 1 .. nz-2; pack_end_planes adds the two end planes), else null
  uint8_t *fusePack = nullptr;
  // test hook: fill fresh cells with one thread in list order
  bool sequentialFill = false;
  int stepBegunNs = -1;
  bool planOfStep = false;  // the device plan is the begun step's
  // no tag has been written since the last step's retag (planes copied from
  // another slab of the scene are that slab's)
  bool tagsOfStep = false;
  // a cell that a step does not update may differ between the halves (a field
  // write, a phase-by-phase call): carried over the whole grid before the next
  // fused step
  bool carrySolid = false;
  int fullRetagSteps = 0;
  int nsphLast = 0;

  // z slab of a larger scene (lbm_set_slab): local plane k is global plane
  // k + zoff; planes [ownLo, ownHi] are this handle's, the others copies of
  // its neighbours' (slab = false: the whole grid is the scene)
  bool slab = false;
  int zoff = 0, ownLo = 0, ownHi = 0;

  int *linkChunks = nullptr;  // generic-solid link compaction: per-chunk counts, then offsets
  long long linkChunksCap = 0;
  void *linkBuf = nullptr;  // the link list (cells, moms, dirs) on the device
  long long linkBufCap = 0;  // links

  size_t deviceBytes = 0;
  long long launches = 0;
  unsigned long long h2dBytes = 0, d2hBytes = 0;
  std::string err;

  // absorbDeadCells computed by the step that precedes it (lbm_step_end)
  // and fetched with the step's impulses: the result, the spheres it was
  // computed for, and the handle's launch and transfer counts, parameters and
  // current half when it was taken.  lbm_absorb_dead_cells returns it while
  // all of these still match; anything that moves device state in between
  // either changes them or clears `valid` itself.
  struct DeadAhead {
    bool valid = false;
    int ns = 0;
    lbm_sphere sp[LBM_MAX_SPHERES];
    double out[LBM_MAX_SPHERES * 6];
    long long launches = 0;
    unsigned long long h2d = 0, d2h = 0;
    lbm_params params;
    int cur = 0;
  } deadAhead;

  // CUDA-event timing of the fused kernel (lbm_fused_timing)
  bool timing = false;
  std::vector<cudaEvent_t> evStart, evStop;
  size_t evUsed = 0;
};

namespace lbm {
// the tile shape a fused launch of `shape` on this handle uses: the
// TMA-staged and L2-prefetch forms need the scene's tensor maps (nx a
// multiple of 16), otherwise the compact form of the same rows
inline int resolve_shape(const lbm_sim *h, int shape) {
  if ((shape & (LBM_FUSED_TMA | LBM_FUSED_L2PF)) && !h->dMaps)
    return shape_rows(shape) | LBM_FUSED_COMPACT | (shape & SHAPE_WIDE);
  return shape;
}
}  // namespace lbm
