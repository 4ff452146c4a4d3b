// The MLP head for wide layers (fp32; included by model.cuh inside namespace stafb, after mlp.cuh): same mathematics as
// k_mlp_fwd / k_mlp_bwd of mlp.cuh, another split of the work.
//
// mlp.cuh gives a warp two atoms and every weight is loaded once per two atoms; at 140 x 140 that makes shared-memory
// loads, one per multiply-add or two, the limit.  Here a block carries a tile of M atoms through all layers.  Its
// vectors lie feature-major in shared memory, [feature][atom] with rows of ml_rs(M) words, and a thread forms 4 atoms x
// 4 outputs (forward) or 4 atoms x 4 inputs (transposed products) of a layer, so that two 16-byte loads feed sixteen
// multiply-adds.
//   forward     Y[j][a]  = sum_i W[i][j] X[i][a]     per i one row of X, one of W
//   transposed  Xo[i][a] = sum_j W[i][j] D[j][a]     four columns of W at a time
//   dL/dW       G[i][j]  = sum_a h[i][a] q[j][a]     thread: 8 inputs x 4 outputs, four atoms at a time
// Row strides are odd multiples of four words: lanes on consecutive rows read 16 bytes each without bank conflicts.
//
// The weight gradients do not go out as atomics: a block writes the sums of its atoms to a row of its own and k_mlp_sum
// adds the rows up (28,000 words per block otherwise, at the L2's rate for atomics a third of the kernel).
#pragma once

// row stride of a [feature][atom] buffer of M atoms (M a multiple of four)
__host__ __device__ constexpr int ml_rs(int M) { return ((M >> 2) | 1) << 2; }

// What the kernels need to know of a layer, in shared memory (formed once per block: the sums over the layers below,
// re-formed from the model's constants wherever they were needed, took 500 cycles per layer and pass).
struct LayerInfo {
  int in, out;  // inputs, outputs
  int pack;     // its words in the packed copy
  int gofs;     // its weights in the species' parameter block of theta / the gradient (from off_w on)
  int hofs;     // its first row among the activations
};
__device__ __forceinline__ void ml_layer_table(const ModelDev& md, int t, LayerInfo* li) {
  if ((int)threadIdx.x < md.n_dense) {
    const int l = threadIdx.x;
    LayerInfo v;
    v.in = md.in_of(t, l); v.out = md.width[l];
    v.pack = 0;
    for (int k = 0; k < l; k++) v.pack += ml_layer_words(md.in_of(t, k), md.width[k]);
    v.gofs = md.w_off(t, l);
    v.hofs = md.h_off(l);
    li[l] = v;
  }
}

__device__ __forceinline__ void ml_st4(float* p, const float (&x)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
}

// ---- dense products of a tile; the caller puts block barriers around them.  The weights pass through a ring of two
// chunks of ML_RING words in shared memory, the next one on its way (cp.async) while this one is used: read in place,
// a block met an L2 latency every four rows.
constexpr int ML_RING = 2816;  // words of a chunk: 16 rows of a 140-wide layer, 16 columns of 140 rows
__host__ __device__ inline int ml_chunk_rows(int ld) { return ML_RING / ld; }                 // forward: whole rows
__host__ __device__ inline int ml_chunk_cols(int in) { return (ML_RING / in - 4) & ~7; }      // transposed: columns
__device__ __forceinline__ void cp16(float* dst, const float* src) { __pipeline_memcpy_async(dst, src, 16); }

// Y[j][a] = act( b[j] + sum_i X[i][a] W[i,j] )
template <int M, bool TANH, bool BIAS>
__device__ __forceinline__ void tile_fwd(int in, int out, const LayerView<float>& lv, const float* __restrict__ X,
                                         float* __restrict__ Y, float* __restrict__ ring) {
  constexpr int RS = ml_rs(M), A4 = M / 4;
  if (out == 1) {  // the energy: four threads per atom
    static_assert(M % 8 == 0, "whole warps");
    const int a = threadIdx.x >> 2, p = threadIdx.x & 3;
    if (a < M) {
      float s = 0.0f;
#pragma unroll 8
      for (int i = p; i < in; i += 4) s += X[i * RS + a] * lv.W[i * lv.ld];
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (BIAS) s += lv.B[0];
      if (p == 0) Y[a] = TANH ? ml_tanh(s) : s;
    }
    return;
  }
  const int nq = ((out + 3) >> 2) * A4, ld = lv.ld, kc = ml_chunk_rows(ld);
  auto fetch = [&](int i0, float* dst) {
    const int words = min(kc, in - i0) * ld;
    for (int x = threadIdx.x * 4; x < words; x += blockDim.x * 4) cp16(dst + x, lv.W + i0 * ld + x);
  };
  for (int qb = 0; qb < nq; qb += blockDim.x) {  // one round unless the layer is wider than the block
    const int q = qb + threadIdx.x, at = q % A4, j0 = (q / A4) * 4;
    const bool mine = q < nq;
    const float* x = X + 4 * at;
    float acc[4][4];
#pragma unroll
    for (int c = 0; c < 4; c++)
#pragma unroll
      for (int a = 0; a < 4; a++) acc[c][a] = 0.0f;
    float bias[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (BIAS && mine) ml_ld4(lv.B + j0, bias);
    fetch(0, ring);
    __pipeline_commit();
    int buf = 0;
    for (int i0 = 0; i0 < in; i0 += kc, buf ^= 1) {
      if (i0 + kc < in) fetch(i0 + kc, ring + (buf ^ 1) * ML_RING);
      __pipeline_commit();
      __pipeline_wait_prior(1);
      __syncthreads();
      if (mine) {
        const float* w = ring + buf * ML_RING + j0;
        const int n = min(kc, in - i0);
#pragma unroll 4
        for (int i = 0; i < n; i++) {
          float xv[4], wv[4];
          ml_ld4(x + (i0 + i) * RS, xv);
          ml_ld4(w + i * ld, wv);
#pragma unroll
          for (int c = 0; c < 4; c++)
#pragma unroll
            for (int a = 0; a < 4; a++) acc[c][a] += wv[c] * xv[a];
        }
      }
      __syncthreads();
    }
    if (mine) {
#pragma unroll
      for (int c = 0; c < 4; c++) {
        if (j0 + c < out) {
#pragma unroll
          for (int a = 0; a < 4; a++) { acc[c][a] += bias[c]; if (TANH) acc[c][a] = ml_tanh(acc[c][a]); }
          ml_st4(Y + (j0 + c) * RS + 4 * at, acc[c]);
        }
      }
    }
  }
}

// Xo[i][a] = sum_j D[j][a] W[i,j]  (and the same for a second cotangent D2 -> Xo2 when TWO)
template <int M, bool TWO>
__device__ __forceinline__ void tile_bwd(int in, int out, const LayerView<float>& lv, const float* __restrict__ D,
                                         float* __restrict__ Xo, const float* __restrict__ D2,
                                         float* __restrict__ Xo2, float* __restrict__ ring) {
  constexpr int RS = ml_rs(M), A4 = M / 4, TI = 4;
  const int ld = lv.ld;
  if (out == 1) {  // the last layer: an outer product
    for (int q = threadIdx.x; q < in * A4; q += blockDim.x) {
      const int i = q / A4, at = q - i * A4;
      const float w = lv.W[i * ld];
      float d[4];
      ml_ld4(D + 4 * at, d);
#pragma unroll
      for (int a = 0; a < 4; a++) d[a] *= w;
      ml_st4(Xo + i * RS + 4 * at, d);
      if (TWO) {
        ml_ld4(D2 + 4 * at, d);
#pragma unroll
        for (int a = 0; a < 4; a++) d[a] *= w;
        ml_st4(Xo2 + i * RS + 4 * at, d);
      }
    }
    return;
  }
  const int ni = (in + TI - 1) / TI, nq = ni * A4, jc = ml_chunk_cols(in), cs = jc + 4, o4 = (out + 3) & ~3;
  auto fetch = [&](int j0, float* dst) {  // columns j0 .. of every row (the padding columns of a row are zero)
    const int n4 = min(jc, o4 - j0) >> 2;
    for (int x = threadIdx.x; x < in * n4; x += blockDim.x) {
      const int i = x / n4, k = x - i * n4;
      cp16(dst + i * cs + 4 * k, lv.W + (size_t)i * ld + j0 + 4 * k);
    }
  };
  for (int qb = 0; qb < nq; qb += blockDim.x) {
    const int q = qb + threadIdx.x, at = q % A4, it = q / A4;
    const bool mine = q < nq;
    int wr[TI];
#pragma unroll
    for (int r = 0; r < TI; r++) {
      const int i = it + r * ni;  // consecutive lanes on consecutive rows
      wr[r] = (i < in ? i : in - 1) * cs;
    }
    float acc[TI][4], acc2[TI][4];
#pragma unroll
    for (int r = 0; r < TI; r++)
#pragma unroll
      for (int a = 0; a < 4; a++) acc[r][a] = acc2[r][a] = 0.0f;
    fetch(0, ring);
    __pipeline_commit();
    int buf = 0;
    for (int j0 = 0; j0 < out; j0 += jc, buf ^= 1) {
      if (j0 + jc < out) fetch(j0 + jc, ring + (buf ^ 1) * ML_RING);
      __pipeline_commit();
      __pipeline_wait_prior(1);
      __syncthreads();
      if (mine) {
        const float* w = ring + buf * ML_RING;
        const int n = min(jc, out - j0);
        for (int j = 0; j < n; j += 4) {
          float wv[TI][4];
#pragma unroll
          for (int r = 0; r < TI; r++) ml_ld4(w + wr[r] + j, wv[r]);
#pragma unroll
          for (int c = 0; c < 4; c++) {
            if (j + c >= n) break;  // only in the last chunk; the rows of D end there
            float d[4];
            ml_ld4(D + (j0 + j + c) * RS + 4 * at, d);
#pragma unroll
            for (int r = 0; r < TI; r++)
#pragma unroll
              for (int a = 0; a < 4; a++) acc[r][a] += wv[r][c] * d[a];
            if (TWO) {
              ml_ld4(D2 + (j0 + j + c) * RS + 4 * at, d);
#pragma unroll
              for (int r = 0; r < TI; r++)
#pragma unroll
                for (int a = 0; a < 4; a++) acc2[r][a] += wv[r][c] * d[a];
            }
          }
        }
      }
      __syncthreads();
    }
    if (mine) {
#pragma unroll
      for (int r = 0; r < TI; r++) {
        const int i = it + r * ni;
        if (i < in) {
          ml_st4(Xo + i * RS + 4 * at, acc[r]);
          if (TWO) ml_st4(Xo2 + i * RS + 4 * at, acc2[r]);
        }
      }
    }
  }
}

// rows of a tile's buffers: forward X | H | two cotangents; backward X | V | H | HD | DQ | DP of every layer | two
// cotangents at the inputs
__host__ __device__ inline int ml_tile_fwd_rows(int Fm, int Hs, int mw) { return Fm + Hs + 2 * mw; }
__host__ __device__ inline int ml_tile_bwd_rows(int Fm, int Hs) { return 4 * Fm + 4 * Hs; }

// How the tiles of a species are dealt to blocks: tiles first, first + nb, ... of species t.
struct TilePlan {
  int nb[STAFB_MAX_TYPES];  // blocks of species t
  __device__ __forceinline__ void locate(const ModelDev& md, int& t, int& first) const {
    first = blockIdx.x;
    t = 0;
    while (t < md.nt - 1 && first >= nb[t]) first -= nb[t++];
  }
};

// Forward: e_i, the activations for the backward kernel (acts) and netderiv = d(sum e)/dAF.
// acts: [tile][Hs][M], tiles in species order.
template <int M, int NT>
__global__ void __launch_bounds__(NT)
    k_mlp_fwd_tile(ModelDev md, int nf, const float* __restrict__ theta, const float* __restrict__ wpack, int wstride,
                   const float* __restrict__ af, float* __restrict__ acts, float* __restrict__ e_atom,
                   float* __restrict__ netderiv) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RS = ml_rs(M);
  __shared__ long long rows[M];
  __shared__ LayerInfo li[STAFB_MAX_DENSE];
  int t, q0;
  locate_block(md, nf, M, t, q0);
  const int nat = nf * md.tipos[t], tid = threadIdx.x;
  const int F = md.Fr[t] + md.Fa[t], Lq = md.n_dense, Fm = md.Fmax, Hs = md.Hsum, mw = md.maxw;
  float* ring = reinterpret_cast<float*>(smem_raw);
  float* X = ring + 2 * ML_RING;                  // [Fm]
  float* H = X + Fm * RS;                         // [Hs]
  float* C0 = H + Hs * RS;                        // [mw]
  float* C1 = C0 + mw * RS;                       // [mw]
  const float* mu = theta + md.off_mu[t];
  const float* wp = wpack + (size_t)t * wstride;
  ml_layer_table(md, t, li);
  if (tid < M) rows[tid] = ml_atom_row(md, t, q0, nat, tid);
  __syncthreads();
  chain_wait();  // the packed weights are older than the preceding kernel; everything read below is its output
  for (int idx = tid; idx < M * F; idx += NT) {  // consecutive threads on consecutive fingerprints of one atom
    const int a = idx / F, i = idx - a * F;
    const long long g = rows[a];
    X[i * RS + a] = g >= 0 ? r_log(af[g * Fm + i] + 1e-3f) - mu[i] : 0.0f;
  }
  __syncthreads();
  const float* hin = X;
  for (int l = 0; l < Lq; l++) {
    const LayerInfo v = li[l];
    const LayerView<float> lv = layer_view<float>(v.in, v.out, wp + v.pack);
    float* hout = H + v.hofs * RS;
    if (l < Lq - 1) tile_fwd<M, true, true>(v.in, v.out, lv, hin, hout, ring);
    else tile_fwd<M, false, true>(v.in, v.out, lv, hin, hout, ring);
    __syncthreads();
    hin = hout;
  }
  if (acts) {
    float* ab = acts + (size_t)blockIdx.x * Hs * M;
    for (int idx = tid; idx < Hs * M; idx += NT) ab[idx] = H[(idx / M) * RS + (idx % M)];
  }
  if (tid < M && rows[tid] >= 0) e_atom[rows[tid]] = hin[tid];  // summed per frame by k_loss
  // de/dx by the reverse sweep: cn = cotangent on the pre-activation of layer l
  float* cn = C0;
  float* cp = C1;
  if (tid < M) cn[tid] = 1.0f;
  __syncthreads();
  for (int l = Lq - 1; l >= 0; l--) {
    const LayerInfo v = li[l];
    const LayerView<float> lv = layer_view<float>(v.in, v.out, wp + v.pack);
    if (l < Lq - 1) {
      const float* hl = H + v.hofs * RS;
      for (int idx = tid; idx < v.out * RS; idx += NT) cn[idx] *= (1.0f - hl[idx] * hl[idx]);
      __syncthreads();
    }
    tile_bwd<M, false>(v.in, v.out, lv, cn, cp, nullptr, nullptr, ring);
    __syncthreads();
    float* tmp = cn; cn = cp; cp = tmp;
  }
  for (int idx = tid; idx < M * Fm; idx += NT) {
    const int a = idx / Fm, i = idx - a * Fm;
    const long long g = rows[a];
    if (g >= 0) netderiv[g * Fm + i] = (i < F) ? cn[i * RS + a] / (af[g * Fm + i] + 1e-3f) : 0.0f;
  }
}

// Weight gradients of all layers over the atoms of a tile, the 8 x 4 tiles (8 inputs x 4 outputs) of all layers numbered
// consecutively and dealt to the threads.  The outputs of a tile are nJ apart, so that consecutive lanes read
// consecutive rows of cotangents and write consecutive words; its inputs are consecutive and (nearly) the same for all
// lanes of a warp.  ADD: onto what the block's row already holds.
template <int M, bool ADD>
__device__ __forceinline__ void tile_dw(const LayerInfo* li, int n, const float* __restrict__ X,
                                        const float* __restrict__ V, const float* __restrict__ H,
                                        const float* __restrict__ HD, const float* __restrict__ DQ,
                                        const float* __restrict__ DP, float* __restrict__ gw) {
  constexpr int RS = ml_rs(M), GI = 8;
  int tot = 0;
  for (int l = 0; l < n; l++) tot += ((li[l].in + GI - 1) / GI) * ((li[l].out + 3) >> 2);
  for (int tile = threadIdx.x; tile < tot; tile += blockDim.x) {
    int l = 0, lt = tile;
    LayerInfo v = li[0];
    while (l < n - 1) {
      const int k = ((v.in + GI - 1) / GI) * ((v.out + 3) >> 2);
      if (lt < k) break;
      lt -= k;
      v = li[++l];
    }
    const int in = v.in, out = v.out, nJ = (out + 3) >> 2;
    const int it = lt / nJ, jt = lt - it * nJ, i0 = it * GI;
    const float* hi = (l == 0) ? X : H + li[l - 1].hofs * RS;
    const float* vi = (l == 0) ? V : HD + li[l - 1].hofs * RS;
    const float* dq = DQ + v.hofs * RS;
    const float* dp = DP + v.hofs * RS;
    int jr[4];
#pragma unroll
    for (int r = 0; r < 4; r++) jr[r] = min(jt + r * nJ, out - 1) * RS;
    float g[GI][4];
#pragma unroll
    for (int r = 0; r < GI; r++)
#pragma unroll
      for (int c = 0; c < 4; c++) g[r][c] = 0.0f;
#pragma unroll 1
    for (int a = 0; a < M; a += 4) {
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const float* h_ = (half ? vi : hi) + a;
        const float* q_ = (half ? dp : dq) + a;
        float qv[4][4];
#pragma unroll
        for (int c = 0; c < 4; c++) ml_ld4(q_ + jr[c], qv[c]);
#pragma unroll
        for (int r = 0; r < GI; r++) {
          float hv[4];
          ml_ld4(h_ + min(i0 + r, in - 1) * RS, hv);
#pragma unroll
          for (int c = 0; c < 4; c++)
#pragma unroll
            for (int e = 0; e < 4; e++) g[r][c] += hv[e] * qv[c][e];
        }
      }
    }
    float* dst = gw + v.gofs + i0 * out + jt;
#pragma unroll
    for (int r = 0; r < GI; r++) {
      if (i0 + r < in)
#pragma unroll
        for (int c = 0; c < 4; c++)
          if (jt + c * nJ < out) {
            float* p = dst + r * out + c * nJ;
            *p = ADD ? *p + g[r][c] : g[r][c];
          }
    }
  }
  // bias gradients: sums of the first-order cotangents
  for (int l = 0; l < n; l++) {
    float* gb = gw + li[l].gofs + li[l].in * li[l].out;
    for (int j = threadIdx.x; j < li[l].out; j += blockDim.x) {
      const float* q = DQ + (li[l].hofs + j) * RS;
      float s = 0.0f;
#pragma unroll
      for (int a = 0; a < M; a++) s += q[a];
      gb[j] = ADD ? gb[j] + s : s;
    }
  }
}

// Backward: see k_mlp_bwd.  part: [block][pstride] sums over the block's atoms in the layout of the species' parameter
// block (k_mlp_sum adds them into the gradient).  A block takes every nb-th tile of its species.
template <int M, int NT>
__global__ void __launch_bounds__(NT)
    k_mlp_bwd_tile(ModelDev md, int nf, const float* __restrict__ theta, const float* __restrict__ wpack, int wstride,
                   const float* __restrict__ af, const float* __restrict__ acts, const float* __restrict__ ebar /*[nf]*/,
                   const float* __restrict__ u /*[nf,N,Fmax]*/, const float* __restrict__ vrow /*[nf,N,nv]*/, int nv,
                   float* __restrict__ gaf, float* __restrict__ part, int pstride, TilePlan tp) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int RS = ml_rs(M);
  __shared__ long long rows[M];
  __shared__ LayerInfo li[STAFB_MAX_DENSE];
  int t, first;
  tp.locate(md, t, first);
  const int nat = nf * md.tipos[t], tid = threadIdx.x, ntile = (nat + M - 1) / M;
  int tile0 = 0;  // tiles of the species before this one (acts' numbering)
  for (int k = 0; k < t; k++) tile0 += (nf * md.tipos[k] + M - 1) / M;
  const int F = md.Fr[t] + md.Fa[t], Lq = md.n_dense, Fm = md.Fmax, Hs = md.Hsum;
  float* ring = reinterpret_cast<float*>(smem_raw);
  float* X = ring + 2 * ML_RING;                  // x
  float* V = X + Fm * RS;                         // tangent on x
  float* H = V + Fm * RS;                         // activations
  float* HD = H + Hs * RS;                        // tangents of the activations
  float* DQ = HD + Hs * RS;                       // cotangents on the pre-activations
  float* DP = DQ + Hs * RS;                       //    and on their tangents
  float* G0 = DP + Hs * RS;                       // cotangents on x
  float* G1 = G0 + Fm * RS;                       //    and v
  const float* mu = theta + md.off_mu[t];
  const float* wp = wpack + (size_t)t * wstride;
  float* my = part + (size_t)blockIdx.x * pstride;
  float* gw = my + (md.off_w[t] - md.off_a2[t]);
  ml_layer_table(md, t, li);
  chain_wait();  // the packed weights are older than the preceding kernel; everything read below is its output
  for (int tl = first; tl < ntile; tl += tp.nb[t]) {
    const bool again = tl != first;
    __syncthreads();  // the sums of the tile before this one are formed
    if (tid < M) rows[tid] = ml_atom_row(md, t, tl * M, nat, tid);
    __syncthreads();
    for (int idx = tid; idx < M * F; idx += NT) {
      const int a = idx / F, i = idx - a * F;
      const long long g = rows[a];
      float xv = 0.0f, vv = 0.0f;
      if (g >= 0) {
        const float den = af[g * Fm + i] + 1e-3f;
        xv = r_log(den) - mu[i];
        vv = u[g * Fm + i] / den;
      }
      X[i * RS + a] = xv;
      V[i * RS + a] = vv;
    }
    {
      const float* ab = acts + (size_t)(tile0 + tl) * Hs * M;
      for (int idx = tid; idx < Hs * M; idx += NT) {
        const int a = idx % M;
        H[(idx / M) * RS + a] = rows[a] >= 0 ? ab[idx] : 0.0f;
      }
    }
    __syncthreads();
    // forward tangent: HD = (HDin W) * act'
    const float* hdin = V;
    for (int l = 0; l < Lq - 1; l++) {
      const LayerInfo v = li[l];
      const LayerView<float> lv = layer_view<float>(v.in, v.out, wp + v.pack);
      float* hdo = HD + v.hofs * RS;
      tile_fwd<M, false, false>(v.in, v.out, lv, hdin, hdo, ring);
      __syncthreads();
      const float* ho = H + v.hofs * RS;
      for (int idx = tid; idx < v.out * RS; idx += NT) hdo[idx] *= (1.0f - ho[idx] * ho[idx]);
      __syncthreads();
      hdin = hdo;
    }
    // reverse over (h, hd): (cq, cp) = cotangents on (h, hd) of the current layer's output, turned into cotangents on
    // the pre-activation and its tangent in place; the last layer is linear
    float* cq = DQ + li[Lq - 1].hofs * RS;
    float* cp = DP + li[Lq - 1].hofs * RS;
    if (tid < M) {
      const long long g = rows[tid];
      cq[tid] = g >= 0 ? ebar[g / md.N] : 0.0f;
      cp[tid] = g >= 0 ? 1.0f : 0.0f;
    }
    __syncthreads();
    for (int l = Lq - 1; l >= 0; l--) {
      const LayerInfo v = li[l];
      const LayerView<float> lv = layer_view<float>(v.in, v.out, wp + v.pack);
      if (l < Lq - 1) {
        const float* ho = H + v.hofs * RS;
        const float* hd = HD + v.hofs * RS;
        for (int idx = tid; idx < v.out * RS; idx += NT) {
          const float hh = ho[idx], d1 = 1.0f - hh * hh, c = cp[idx];
          cp[idx] = c * d1;
          cq[idx] = cq[idx] * d1 - 2.0f * hh * hd[idx] * c;
        }
        __syncthreads();
      }
      float* nq = l > 0 ? DQ + li[l - 1].hofs * RS : G0;  // of the layer below (or of x, v)
      float* np = l > 0 ? DP + li[l - 1].hofs * RS : G1;
      tile_bwd<M, true>(v.in, v.out, lv, cq, nq, cp, np, ring);
      __syncthreads();
      cq = nq;
      cp = np;
    }
    if (again) tile_dw<M, true>(li, Lq, X, V, H, HD, DQ, DP, gw);
    else tile_dw<M, false>(li, Lq, X, V, H, HD, DQ, DP, gw);
    // G0 = dS/dx, G1 = dS/dv  ->  dL/dmu; dL/dAF, also kept in place of G1 for the contraction below
    for (int i = tid; i < F; i += NT) {
      float s = 0.0f;
#pragma unroll
      for (int a = 0; a < M; a++) s -= G0[i * RS + a];
      float* p = my + (md.off_mu[t] - md.off_a2[t]) + i;
      *p = again ? *p + s : s;
    }
    for (int idx = tid; idx < M * Fm; idx += NT) {
      const int a = idx / Fm, i = idx - a * Fm;
      const long long g = rows[a];
      float v = 0.0f;
      if (g >= 0 && i < F) {
        const float den = af[g * Fm + i] + 1e-3f;
        v = G0[i * RS + a] / den + G1[i * RS + a] * (-u[g * Fm + i] / (den * den));
      }
      if (g >= 0) gaf[g * Fm + i] = v;
      if (i < F) G1[i * RS + a] = v;
    }
    __syncthreads();
    // dL/dalpha (fingerprint part) = sum_atoms dL/dAF[c(q)] * dAF[c(q)]/dalpha[q]; alpha2b and alpha3b
    // are contiguous in theta, q runs over both
    const int Fr = md.Fr[t], Fa = md.Fa[t], n2 = md.nt * Fr, nq = n2 + md.C * 3 * Fa;
    for (int q = tid; q < nq; q += NT) {
      const int ch = q < n2 ? (q % Fr) : Fr + ((q - n2) / 3) % Fa;
      // position of parameter q in the rows the fingerprint sweep wrote: its accumulator layout
      // alpha2b[nt,Frmax] | alpha3b[C,3*Famax] (equal to q when every species has the same channel counts)
      int qa;
      if (q < n2) qa = (q / Fr) * md.Frmax + (q % Fr);
      else {
        const int r = q - n2, sc = r / 3, s = sc / Fa;
        qa = md.nt * md.Frmax + (s * md.Famax + (sc - s * Fa)) * 3 + (r - sc * 3);
      }
      float g = 0.0f;
#pragma unroll 8
      for (int a = 0; a < M; a++) {
        const long long r = rows[a];
        if (r >= 0) g += G1[ch * RS + a] * vrow[r * nv + qa];
      }
      my[q] = again ? my[q] + g : g;
    }
  }
}

// Adds the rows of sums that k_mlp_bwd_tile left: grad += sum over the species' blocks.  A block of 256 threads takes 32
// consecutive parameters, eight threads each over every eighth row (coalesced 128-byte reads, many in flight).
static __global__ void __launch_bounds__(256)
    k_mlp_sum(ModelDev md, TilePlan tp, const float* __restrict__ part, int pstride, float* __restrict__ grad,
              int n_params) {
  __shared__ float red[8][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int p = blockIdx.x * 32 + lane;
  int t = 0, b0 = 0;
  if (p < n_params)
    while (t < md.nt - 1 && p >= md.off_a2[t + 1]) b0 += tp.nb[t++];
  chain_wait();
  float s = 0.0f;
  if (p < n_params) {
    const float* src = part + (size_t)b0 * pstride + (p - md.off_a2[t]);
    const int nb = tp.nb[t];
#pragma unroll 4
    for (int k = w; k < nb; k += 8) s += src[(size_t)k * pstride];
  }
  red[w][lane] = s;
  __syncthreads();
  if (w == 0 && p < n_params) {
#pragma unroll
    for (int k = 1; k < 8; k++) s += red[k][lane];
    grad[p] += s;
  }
}
