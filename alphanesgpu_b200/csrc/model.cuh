// The model handle of the fused path and what its translation units share: fused.cu (housekeeping, loss, Adam, entry
// points), sweep_f32.cu / sweep_f64.cu (the sweeps) and mlp_f32.cu / mlp_f64.cu (the network kernels).
#pragma once
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include <type_traits>
#include "common.cuh"

namespace stafb {

constexpr int ML_THREADS = 256;

struct ModelDev {
  int nt, C, N, ncls;
  int tipos[STAFB_MAX_TYPES], shift[STAFB_MAX_TYPES + 1], Fr[STAFB_MAX_TYPES], Fa[STAFB_MAX_TYPES];
  int off_a2[STAFB_MAX_TYPES], off_a3[STAFB_MAX_TYPES], off_mu[STAFB_MAX_TYPES], off_w[STAFB_MAX_TYPES];
  int off_emb[STAFB_MAX_TYPES];
  int n_dense, width[STAFB_MAX_DENSE];
  int Fmax, Frmax, Famax, Hsum, maxw;
  __host__ __device__ int in_of(int t, int l) const { return l == 0 ? Fr[t] + Fa[t] : width[l - 1]; }
  __host__ __device__ int w_off(int t, int l) const {
    int s = 0;
    for (int k = 0; k < l; k++) s += in_of(t, k) * width[k] + width[k];
    return s;
  }
  __host__ __device__ int h_off(int l) const {  // offset of the output of Dense l in the activation row
    int s = 0;
    for (int k = 0; k < l; k++) s += width[k];
    return s;
  }
  __host__ __device__ int type_of(int id) const {
    int t = 0;
    while (t < nt - 1 && id >= shift[t + 1]) t++;
    return t;
  }
};

// species-major enumeration: block -> (species t, index q0 of its first atom among the nf*tipos[t]
// atoms of that species); W atoms per block, blocks never mix species
__device__ __forceinline__ void locate_block(const ModelDev& md, int nf, int W, int& t, int& q0) {
  int blk = blockIdx.x;
  t = 0;
  while (t < md.nt - 1) {
    const int nb = (nf * md.tipos[t] + W - 1) / W;
    if (blk < nb) break;
    blk -= nb;
    t++;
  }
  q0 = blk * W;
}

__device__ __forceinline__ bool locate_atom(const ModelDev& md, int nf, int W, int slot, int& t, int& b, int& i) {
  int q0;
  locate_block(md, nf, W, t, q0);
  const int q = q0 + slot;
  if (q >= nf * md.tipos[t]) return false;
  b = q / md.tipos[t];
  i = md.shift[t] + (q - b * md.tipos[t]);
  return true;
}

static inline int species_blocks(const ModelDev& md, int nf, int W) {
  int s = 0;
  for (int t = 0; t < md.nt; t++) s += (nf * md.tipos[t] + W - 1) / W;
  return s;
}

#include "devmath.cuh"
#include "sweep.cuh"

// ---------------------------------------------------------------------------- MLP head
#include "mlp.cuh"
#include "mlp_tile.cuh"
#include "mlp_mma.cuh"

}  // namespace stafb

using namespace stafb;

struct stafb_model {
  stafb_ctx* ctx;
  ModelDev md;
  int n_params, n_emb;
  int blk_size[STAFB_MAX_TYPES];
  size_t es;
  int cap_atoms;  // atoms per frame the scratch was sized for
  int aw;   // atoms per warp of the MLP kernels (4, 2 or 1; a block of eight warps owns 8*aw atoms)
  int stage;  // Dense layers in shared memory: 2 all at kernel start, 1 one at a time, 0 none
  int tile_above;  // the tile form of the MLP kernels (mlp_tile.cuh) takes evaluations of more 16-atom blocks; -1: none
  void* part;  // rows of gradient sums of its backward kernel [part_blocks][part_stride]
  int part_blocks, part_stride;
  size_t mlp_fwd_smem, mlp_bwd_smem;
  // scratch for max_batch frames
  void *rows, *af, *nd, *acts, *e_atom, *force, *flab, *ebar, *gradnet, *gaf, *energy, *vrow;
  int row_stride;      // bytes per neighbour record (common.cuh)
  unsigned char* spar;  // per-species parameter blocks of the sweeps, rewritten by k_prep at every evaluation
  SparLayout sl;
  void* wpack;  // packed, padded Dense layers of every species (k_prep), wstride elements per species
  int wstride;
  int nv;  // row length of vrow: nt*Frmax + C*3*Famax
  // tensor-core MLP kernels (fp32): on/off, warps per block (16 atoms), the fragment-ordered pack and its
  // per-species stride, dynamic shared memory of the two kernels
  int mma, mma_nw, mma_stage, wm_stride;
  void* wm;
  size_t mma_fwd_smem, mma_bwd_smem;
  double* epart;     // partial energy sums of k_loss: [nf][eb]; from [max_batch][LOSS_EB_MAX] on: one arrival counter per frame
  double* losses_d;  // [0..4] the four losses + the done-counter of k_loss; [8 + b] sum of the atomic energies of
                     // frame b (accumulated by the MLP kernel); from [8 + max_batch] on the virial accumulators [b][9][VIR_SLOTS]
  // staging for the *_host entry points
  // two pipelined slots for stafb_train_step_host_begin/_end: pinned input block (pos | f_label | box | e_label),
  // pinned results (4 losses + status) and the event that marks the slot's step complete
  char* slot_in_h[3];  // slots 0, 1: the pipelined calls; slot 2: the synchronous stafb_train_step_host
  double* slot_out_h[3];
  cudaEvent_t slot_done[3];
  int slot_busy[3];
  // per slot: the captured graph of (copy in, step, copy out) and the call signature it was captured for
  struct SlotKey {
    int nf, loss_kind;
    const void *theta, *emb, *grad, *stream;
    double pe, pf, pb, bound, pv;
    int with_v;
  } slot_key[3];
  double* mirror_next;  // mapped host memory the next training evaluation's k_loss writes its results to
  void* vlab_d;         // device copy of the virial labels of a host-buffer step [max_batch][9]
  int slot_state[3];  // 0: nothing yet, 1: signature seen once (ran eagerly), 2: graph instantiated, -1: capture failed
  cudaGraphExec_t slot_exec[3];
  // Two more sets of neighbour rows (a context of their own for the search scratch + the compact rows), so that
  // the geometry of the NEXT step, which depends on no trainable parameter, can be built on another stream while
  // this step's sweeps still read theirs.  Allocated on first use.
  struct NlSet {
    stafb_ctx* ctx;
    void* rows;
    cudaEvent_t ready;
    int nf;  // frames the set currently describes (0: nothing)
  } nl[2];
  cudaStream_t side;  // stream of the prefetches issued by stafb_train_step_host_begin
  cudaGraphExec_t nl_exec[2];
  size_t smem_limit;
};

// words of shared memory the staged Dense layers need: stage 1 = the largest (in + 1) x row stride over the
// layers, stage 2 = all layers of one species back to back
static size_t mlp_stage_words(const ModelDev& d, int stage) {
  size_t best = 0;
  for (int t = 0; t < d.nt; t++) {
    size_t sum = 0;
    for (int l = 0; l < d.n_dense; l++) {
      const size_t wds = (size_t)(d.in_of(t, l) + 1) * ml_ld(d.width[l]);
      sum += wds;
      if (stage == 1) best = wds > best ? wds : best;
    }
    if (stage == 2) best = sum > best ? sum : best;
  }
  return stage ? best : 0;
}
static size_t mlp_smem_fwd(const ModelDev& d, size_t es, int aw, int stage) {
  return es * (ML_WARPS * ml_fwd_words(d.Fmax, d.Hsum, d.maxw, aw) + mlp_stage_words(d, stage));
}
static size_t mlp_smem_bwd(const ModelDev& d, size_t es, int aw, int stage) {
  return es * (ML_WARPS * ml_bwd_words(d.Fmax, d.Hsum, d.maxw, aw) + mlp_stage_words(d, stage));
}

constexpr int ML_TILE = 24, ML_TILE_THREADS = 384;
static size_t mlp_tile_smem_fwd(const ModelDev& d, int tile) {
  return sizeof(float) * (2 * ML_RING + (size_t)ml_tile_fwd_rows(d.Fmax, d.Hsum, d.maxw) * ml_rs(tile));
}
static size_t mlp_tile_smem_bwd(const ModelDev& d, int tile) {
  return sizeof(float) * (2 * ML_RING + (size_t)ml_tile_bwd_rows(d.Fmax, d.Hsum) * ml_rs(tile));
}
// Which form of the MLP kernels an evaluation of nf frames takes: see stafb_model_create.
static bool mlp_tiles(const stafb_model* m, int nf) {
  return m->tile_above >= 0 && species_blocks(m->md, nf, 16) > m->tile_above;
}
// blocks of the tile form's backward kernel: one per tile, at most `slots` in all, shared out by the species' tiles
static TilePlan mlp_tile_plan(const ModelDev& d, int nf, int tile, int slots) {
  TilePlan p = {};
  long long total = 0;
  for (int t = 0; t < d.nt; t++) total += ((long long)nf * d.tipos[t] + tile - 1) / tile;
  for (int t = 0; t < d.nt; t++) {
    const long long n = ((long long)nf * d.tipos[t] + tile - 1) / tile;
    const long long mine = total <= slots ? n : n * (slots - d.nt) / total + 1;
    p.nb[t] = (int)(mine < n ? mine : n);
  }
  return p;
}

// cudaFuncSetAttribute applies to the device that is current when it is called, and one process may drive
// several GPUs (staf_load honours StafOptions.device_id; stafb_peer_connect_local exists for that use): the
// "already opted in" notes of the launchers below are therefore kept per device, as the reference keeps its
// per-device context map (STAF/src/descriptor_builder/reforce.cc:143-158).
constexpr int MAX_DEVICES = 64;
static inline int device_slot() {
  int d = 0;
  cudaGetDevice(&d);
  return (d >= 0 && d < MAX_DEVICES) ? d : 0;
}

// multiprocessors of the current device
static inline int sm_count() {
  int d = 0, n = 148;
  cudaGetDevice(&d);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, d);
  return n;
}

// what a sweep launch needs besides the model: the records of this evaluation and the per-call buffers
template <class T>
struct SweepCall {
  const void* rows;
  int nf, nall;
  const T* chan_in;
  const T* force;  // force-backward sweep: the forces, their labels and the loss's scale (dL/dF is formed on the fly)
  const T* flab;
  T fscale;
  int loss_kind;
  T* out;
  T* grad;
  T* vout;
  double* vir;
  const double* vacc;  // force backward with a virial loss: the virials, their labels, the loss's scale
  const T* vlab;
  T vscale;
  int* status;
};

template <class T, int MODE>
int launch_sweep(stafb_model* m, cudaStream_t s, const SweepCall<T>& call);
template <class T>
int launch_mlp_fwd(stafb_model* m, cudaStream_t s, int nf, const T* theta, const T* af, T* acts, T* e_atom, T* nd);
template <class T>
int launch_mlp_bwd(stafb_model* m, cudaStream_t s, int nf, const T* theta, const T* af, const T* acts, const T* ebar,
                   const T* u, T* gaf, T* grad);
