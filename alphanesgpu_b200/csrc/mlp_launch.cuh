// Launches of the network kernels (mlp.cuh, mlp_mma.cuh), instantiated for REAL by mlp_f32.cu and mlp_f64.cu.
#include "model.cuh"

template <class T, int AW, bool WG, bool WIDE>
static int launch_mlp_fwd_t(stafb_model* m, cudaStream_t s, int nf, const T* theta, const T* af, T* acts, T* e_atom,
                            T* nd) {
  static size_t attr_dev[MAX_DEVICES] = {0};  // largest dynamic shared-memory size opted in for, per device
  size_t& attr = attr_dev[device_slot()];
  if (m->mlp_fwd_smem > 48 * 1024 && m->mlp_fwd_smem > attr) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_mlp_fwd<T, AW, WG, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)m->mlp_fwd_smem));
    attr = m->mlp_fwd_smem;
  }
  STAFB_CUDA_OK(launch_chained(k_mlp_fwd<T, AW, WG, WIDE>, species_blocks(m->md, nf, ML_WARPS * AW), ML_THREADS,
                               m->mlp_fwd_smem, s, m->md, nf, theta, (const T*)m->wpack, m->wstride, af, acts, e_atom,
                               nd, m->stage, (int)mlp_stage_words(m->md, m->stage)));
  m->ctx->launches++;
  return STAFB_OK;
}

template <class T, int AW, bool WG, bool WIDE>
static int launch_mlp_bwd_t(stafb_model* m, cudaStream_t s, int nf, const T* theta, const T* af, const T* acts,
                            const T* ebar, const T* u, T* gaf, T* grad) {
  static size_t attr_dev[MAX_DEVICES] = {0};
  size_t& attr = attr_dev[device_slot()];
  const T* vrow = (const T*)m->vrow;
  if (m->mlp_bwd_smem > 48 * 1024 && m->mlp_bwd_smem > attr) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_mlp_bwd<T, AW, WG, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)m->mlp_bwd_smem));
    attr = m->mlp_bwd_smem;
  }
  STAFB_CUDA_OK(launch_chained(k_mlp_bwd<T, AW, WG, WIDE>, species_blocks(m->md, nf, ML_WARPS * AW), ML_THREADS,
                               m->mlp_bwd_smem, s, m->md, nf, theta, (const T*)m->wpack, m->wstride, af, acts, ebar, u,
                               vrow, m->nv, gaf, grad, m->stage, (int)mlp_stage_words(m->md, m->stage)));
  m->ctx->launches++;
  return STAFB_OK;
}

static int launch_mlp_fwd_tile(stafb_model* m, cudaStream_t s, int nf, const float* theta, const float* af, float* acts,
                               float* e_atom, float* nd) {
  const size_t sm = mlp_tile_smem_fwd(m->md, ML_TILE);
  static size_t attr_dev[MAX_DEVICES] = {0};
  size_t& attr = attr_dev[device_slot()];
  if (sm > 48 * 1024 && sm > attr) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_mlp_fwd_tile<ML_TILE, ML_TILE_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    attr = sm;
  }
  STAFB_CUDA_OK(launch_chained(k_mlp_fwd_tile<ML_TILE, ML_TILE_THREADS>, species_blocks(m->md, nf, ML_TILE), ML_TILE_THREADS, sm, s, m->md, nf, theta,
                               (const float*)m->wpack, m->wstride, af, acts, e_atom, nd));
  m->ctx->launches++;
  return STAFB_OK;
}

static int launch_mlp_bwd_tile(stafb_model* m, cudaStream_t s, int nf, const float* theta, const float* af,
                               const float* acts, const float* ebar, const float* u, float* gaf, float* grad) {
  const size_t sm = mlp_tile_smem_bwd(m->md, ML_TILE);
  static size_t attr_dev[MAX_DEVICES] = {0};
  size_t& attr = attr_dev[device_slot()];
  if (sm > 48 * 1024 && sm > attr) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_mlp_bwd_tile<ML_TILE, ML_TILE_THREADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    attr = sm;
  }
  const TilePlan tp = mlp_tile_plan(m->md, nf, ML_TILE, m->part_blocks);
  int blocks = 0;
  for (int t = 0; t < m->md.nt; t++) blocks += tp.nb[t];
  STAFB_CUDA_OK(launch_chained(k_mlp_bwd_tile<ML_TILE, ML_TILE_THREADS>, blocks, ML_TILE_THREADS, sm, s, m->md, nf, theta, (const float*)m->wpack,
                               m->wstride, af, acts, ebar, u, (const float*)m->vrow, m->nv, gaf, (float*)m->part,
                               m->part_stride, tp));
  STAFB_CUDA_OK(launch_chained(k_mlp_sum, (m->n_params + 31) / 32, 256, 0, s, m->md, tp, (const float*)m->part,
                               m->part_stride, grad, m->n_params));
  m->ctx->launches += 2;
  return STAFB_OK;
}

static int launch_mlp_fwd_mma(stafb_model* m, cudaStream_t s, int nf, const float* theta, const float* af, float* acts,
                              float* e_atom, float* nd) {
  static size_t attr_dev[MAX_DEVICES] = {0};
  size_t& attr = attr_dev[device_slot()];
  if (m->mma_fwd_smem > 48 * 1024 && m->mma_fwd_smem > attr) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_mlp_fwd_mma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)m->mma_fwd_smem));
    attr = m->mma_fwd_smem;
  }
  STAFB_CUDA_OK(launch_chained(k_mlp_fwd_mma, species_blocks(m->md, nf, MM_ATOMS), 32 * m->mma_nw, m->mma_fwd_smem, s,
                               m->md, nf, theta, (const float*)m->wm, m->wm_stride, af, acts, e_atom, nd));
  m->ctx->launches++;
  return STAFB_OK;
}

static int launch_mlp_bwd_mma(stafb_model* m, cudaStream_t s, int nf, const float* theta, const float* af,
                              const float* acts, const float* ebar, const float* u, float* gaf, float* grad) {
  static size_t attr_dev[MAX_DEVICES] = {0};
  size_t& attr = attr_dev[device_slot()];
  if (m->mma_bwd_smem > 48 * 1024 && m->mma_bwd_smem > attr) {
    STAFB_CUDA_OK(cudaFuncSetAttribute(k_mlp_bwd_mma, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)m->mma_bwd_smem));
    attr = m->mma_bwd_smem;
  }
  STAFB_CUDA_OK(launch_chained(k_mlp_bwd_mma, species_blocks(m->md, nf, MM_ATOMS), 32 * m->mma_nw, m->mma_bwd_smem, s,
                               m->md, nf, theta, (const float*)m->wm, m->wm_stride, af, acts, ebar, u,
                               (const float*)m->vrow, m->nv, gaf, grad));
  m->ctx->launches++;
  return STAFB_OK;
}

template <class T>
int launch_mlp_fwd(stafb_model* m, cudaStream_t s, int nf, const T* theta, const T* af, T* acts, T* e_atom,
                          T* nd) {
  if constexpr (std::is_same<T, float>::value) {
    if (m->mma) return launch_mlp_fwd_mma(m, s, nf, theta, af, acts, e_atom, nd);
    if (mlp_tiles(m, nf)) return launch_mlp_fwd_tile(m, s, nf, theta, af, acts, e_atom, nd);
  }
  const bool wg = m->stage == 0, wide = m->md.maxw > 64;  // the dense products' form: see mlp.cuh
  switch (m->aw) {
    case 4: return wg ? (wide ? launch_mlp_fwd_t<T, 4, true, true>(m, s, nf, theta, af, acts, e_atom, nd) : launch_mlp_fwd_t<T, 4, true, false>(m, s, nf, theta, af, acts, e_atom, nd))
                      : (wide ? launch_mlp_fwd_t<T, 4, false, true>(m, s, nf, theta, af, acts, e_atom, nd) : launch_mlp_fwd_t<T, 4, false, false>(m, s, nf, theta, af, acts, e_atom, nd));
    case 2: return wg ? (wide ? launch_mlp_fwd_t<T, 2, true, true>(m, s, nf, theta, af, acts, e_atom, nd) : launch_mlp_fwd_t<T, 2, true, false>(m, s, nf, theta, af, acts, e_atom, nd))
                      : (wide ? launch_mlp_fwd_t<T, 2, false, true>(m, s, nf, theta, af, acts, e_atom, nd) : launch_mlp_fwd_t<T, 2, false, false>(m, s, nf, theta, af, acts, e_atom, nd));
    default: return wg ? (wide ? launch_mlp_fwd_t<T, 1, true, true>(m, s, nf, theta, af, acts, e_atom, nd) : launch_mlp_fwd_t<T, 1, true, false>(m, s, nf, theta, af, acts, e_atom, nd))
                       : (wide ? launch_mlp_fwd_t<T, 1, false, true>(m, s, nf, theta, af, acts, e_atom, nd) : launch_mlp_fwd_t<T, 1, false, false>(m, s, nf, theta, af, acts, e_atom, nd));
  }
}

template <class T>
int launch_mlp_bwd(stafb_model* m, cudaStream_t s, int nf, const T* theta, const T* af, const T* acts,
                          const T* ebar, const T* u, T* gaf, T* grad) {
  if constexpr (std::is_same<T, float>::value) {
    if (m->mma) return launch_mlp_bwd_mma(m, s, nf, theta, af, acts, ebar, u, gaf, grad);
    if (mlp_tiles(m, nf)) return launch_mlp_bwd_tile(m, s, nf, theta, af, acts, ebar, u, gaf, grad);
  }
  const bool wg = m->stage == 0, wide = m->md.maxw > 64;  // the dense products' form: see mlp.cuh
  switch (m->aw) {
    case 4: return wg ? (wide ? launch_mlp_bwd_t<T, 4, true, true>(m, s, nf, theta, af, acts, ebar, u, gaf, grad) : launch_mlp_bwd_t<T, 4, true, false>(m, s, nf, theta, af, acts, ebar, u, gaf, grad))
                      : (wide ? launch_mlp_bwd_t<T, 4, false, true>(m, s, nf, theta, af, acts, ebar, u, gaf, grad) : launch_mlp_bwd_t<T, 4, false, false>(m, s, nf, theta, af, acts, ebar, u, gaf, grad));
    case 2: return wg ? (wide ? launch_mlp_bwd_t<T, 2, true, true>(m, s, nf, theta, af, acts, ebar, u, gaf, grad) : launch_mlp_bwd_t<T, 2, true, false>(m, s, nf, theta, af, acts, ebar, u, gaf, grad))
                      : (wide ? launch_mlp_bwd_t<T, 2, false, true>(m, s, nf, theta, af, acts, ebar, u, gaf, grad) : launch_mlp_bwd_t<T, 2, false, false>(m, s, nf, theta, af, acts, ebar, u, gaf, grad));
    default: return wg ? (wide ? launch_mlp_bwd_t<T, 1, true, true>(m, s, nf, theta, af, acts, ebar, u, gaf, grad) : launch_mlp_bwd_t<T, 1, true, false>(m, s, nf, theta, af, acts, ebar, u, gaf, grad))
                       : (wide ? launch_mlp_bwd_t<T, 1, false, true>(m, s, nf, theta, af, acts, ebar, u, gaf, grad) : launch_mlp_bwd_t<T, 1, false, false>(m, s, nf, theta, af, acts, ebar, u, gaf, grad));
  }
}

template int launch_mlp_fwd<REAL>(stafb_model*, cudaStream_t, int, const REAL*, const REAL*, REAL*, REAL*, REAL*);
template int launch_mlp_bwd<REAL>(stafb_model*, cudaStream_t, int, const REAL*, const REAL*, const REAL*, const REAL*,
                                  const REAL*, REAL*, REAL*);
