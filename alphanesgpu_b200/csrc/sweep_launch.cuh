// Launches of the sweeps (sweep.cuh), instantiated for REAL by sweep_f32.cu and sweep_f64.cu.
#include "model.cuh"

template <class T, int MODE, int NW, bool PACK = false>
static int launch_sweep_nw(stafb_model* m, cudaStream_t s, const SweepCall<T>& call) {
  const ModelDev& d = m->md;
  const int nr = m->ctx->nr;
  const SweepSmem L = sweep_smem<T>(d, m->sl, nr, MODE, NW, PACK);
  const size_t sm = (size_t)L.total;
  if (sm > m->smem_limit) return STAFB_ERR_CAPACITY;
  constexpr bool F = MODE == MODE_FORCE;
  static bool attr_dev[MAX_DEVICES] = {false};  // per instantiation (T, MODE, NW, PACK) and device
  bool& attr_done = attr_dev[device_slot()];
  if (sm > 48 * 1024 && !attr_done) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_sweep<T, MODE, false, NW, PACK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)m->smem_limit));
    if (F)
      STAFB_CUDA_OK(cudaFuncSetAttribute(k_sweep<T, MODE, F, NW, PACK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)m->smem_limit));
    attr_done = true;
  }
  SweepArgs<T> a;
  a.rows = static_cast<const unsigned char*>(call.rows);
  a.row_stride = m->row_stride;
  a.nr = nr; a.nf = call.nf; a.nall = call.nall;
  a.spar = m->spar;
  a.spar_stride = m->sl.total;
  a.sl = m->sl;
  a.chan_in = call.chan_in; a.force = call.force; a.flab = call.flab; a.fscale = call.fscale;
  a.loss_kind = call.loss_kind; a.out = call.out; a.grad = call.grad;
  a.vout = call.vout; a.nv = m->nv; a.vir = call.vir; a.status = call.status;
  a.vacc = call.vacc; a.vlab = call.vlab; a.vscale = call.vscale;
  const int blocks = call.nf * d.N;
  if (F && call.vir)
    STAFB_CUDA_OK(launch_chained(k_sweep<T, MODE, F, NW, PACK>, blocks, 32 * NW, sm, s, d, a, L));
  else
    STAFB_CUDA_OK(launch_chained(k_sweep<T, MODE, false, NW, PACK>, blocks, 32 * NW, sm, s, d, a, L));
  m->ctx->launches++;
  return STAFB_OK;
}

template <class T, int MODE>
int launch_sweep(stafb_model* m, cudaStream_t s, const SweepCall<T>& call) {
  // Four warps per atom while that still leaves the chip room: a warp alone takes 10-14 us for its atom whatever the
  // others do, and up to about three atoms per SM (two in double precision) the SMs are nearly empty.  Train step of
  // 96 / 300 / 450 atoms: fp32 97 -> 88, 103 -> 97, 110 -> 105 us, fp64 133 -> 112, 141 -> 140, 154 -> 154 us; at 768
  // atoms one warp per atom is the faster form (119 against 141 us).
  static const int few = (sizeof(T) == 4 ? 3 : 2) * sm_count();
  const bool small = call.nf * m->md.N <= few;
  if constexpr (MODE == MODE_FORCE && sizeof(T) == 4) {
    // FP_CH channels per class or fewer on average: partner pairs
    if (m->md.Famax <= FP_CH * m->md.ncls)
      return small ? launch_sweep_nw<T, MODE, 4, true>(m, s, call) : launch_sweep_nw<T, MODE, 1, true>(m, s, call);
  }
  if (small) return launch_sweep_nw<T, MODE, 4>(m, s, call);
  return launch_sweep_nw<T, MODE, 1>(m, s, call);
}

template int launch_sweep<REAL, MODE_AF>(stafb_model*, cudaStream_t, const SweepCall<REAL>&);
template int launch_sweep<REAL, MODE_AFV>(stafb_model*, cudaStream_t, const SweepCall<REAL>&);
template int launch_sweep<REAL, MODE_FORCE>(stafb_model*, cudaStream_t, const SweepCall<REAL>&);
template int launch_sweep<REAL, MODE_FGRAD>(stafb_model*, cudaStream_t, const SweepCall<REAL>&);
