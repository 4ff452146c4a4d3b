// The reference's fingerprint / force / gradient operators on materialised descriptor tensors
// (the drop-in operator boundary).  Arithmetic follows
//   STAF/src/fingerprint/{rad,ang}/reforce.cu.cc, STAF/src/force/{rad,ang}/reforce.cu.cc,
//   STAF/src/grad_finger/{rad,ang}/reforce.cu.cc, STAF/src/grad_force/{rad,ang}/reforce.cu.cc
// of the reference; the execution plan does not: one warp (radial) or one block (angular)
// owns a central atom, reduces in registers / shared memory, and touches global memory with
// one write per output element (per-atom outputs) or one atomic per block (parameter
// gradients) instead of one global atomic per (neighbour, channel).  Channel/class pairs whose
// squared embedding is exactly zero are skipped (they contribute exactly zero).
//
// Angular operators.  The neighbours are grouped by species, so that the triplets of a species-pair class are a
// rectangle (or a triangle) of group members with one parameter row, and the triplet's slot in the caller's tensors
// follows from the two sorted positions.  exp(a1 sj + a2 sk) is a product of table entries exp(a1 s), exp(a2 s) per
// (neighbour, channel), which leaves one exponential per (triplet, channel) instead of three; a chunk of channels
// shares one pass over a class, and its sums one reduction at the end.  What bounds them is the latency of a block's
// passes (staging, tables, triplets, reduction) at one block per atom: 768 atoms, fp32, all central species,
// fingerprints 71 -> 25 us, their gradient 81 -> 28 us, forces 128 -> 41 us, gradient of the forces 92 -> 45 us (the
// form before this one: three library exponentials per (triplet, channel), a block reduction per channel and class,
// and shared-memory float atomics for the forces, whose 32 lanes met on one address).
#include "common.cuh"

namespace stafb {

#include "devmath.cuh"

constexpr int OPS_THREADS = 128;
constexpr int OPS_WARPS = OPS_THREADS / 32;
constexpr int ANG_THREADS = 256;
constexpr int ANG_WARPS = ANG_THREADS / 32;
constexpr int ANG_CH = 8;  // channels per pass at most

__device__ __forceinline__ float op_exp(float x, const float*) { return expf(x); }
__device__ __forceinline__ double op_exp(double x, const double* et) { return exp_table16(x, et); }

// Zero-fills ahead of the operators that accumulate: two buffers, sizes in 4-byte words.  The operator behind it is
// its programmatic dependent and stages its inputs meanwhile.
__global__ void k_zero(int* __restrict__ a, size_t na, int* __restrict__ b, size_t nb) {
  chain_wait();
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x, st = (size_t)gridDim.x * blockDim.x;
  for (size_t q = t; q < na; q += st) a[q] = 0;
  for (size_t q = t; q < nb; q += st) b[q] = 0;
}
static cudaError_t zero_two(cudaStream_t s, void* a, size_t na, void* b, size_t nb) {
  const size_t w = (na > nb ? na : nb) / 4;
  const int blocks = (int)((w + 255) / 256 < 1 ? 1 : ((w + 255) / 256 > 592 ? 592 : (w + 255) / 256));
  return launch_chained(k_zero, blocks, 256, 0, s, (int*)a, na / 4, (int*)b, nb / 4);
}

// Extra inputs / outputs of the ...Virial and ...VirialGrad operators (null pointers: plain operator).
template <class T>
struct VirArgs {
  const T* pos = nullptr;   // [nf,3N] Cartesian positions
  const T* box = nullptr;   // [nf,6]
  T* virial = nullptr;      // force ops: [nf,9] accumulated, W_ab -= g_a r_b
  const T* wbar = nullptr;  // grad ops: [nf,9] cotangent on the virial
};

// r_i - r_j with the minimum image taken in fractional space, as the reference's virial kernels form it
// (STAF/include/staf_force_pbc.cuh:15-49)
template <class T>
__device__ __forceinline__ void mic_cart(const T* __restrict__ pi, const T* __restrict__ pj, const T* __restrict__ B,
                                         T* d) {
  const T i0 = T(1.) / B[0], i1 = -B[1] / (B[0] * B[3]);
  const T i2 = (B[1] * B[4]) / (B[0] * B[3] * B[5]) - B[2] / (B[0] * B[5]);
  const T i3 = T(1.) / B[3], i4 = -B[4] / (B[3] * B[5]), i5 = T(1.) / B[5];
  T rx = (i0 * pi[0] + i1 * pi[1] + i2 * pi[2]) - (i0 * pj[0] + i1 * pj[1] + i2 * pj[2]);
  T ry = (i3 * pi[1] + i4 * pi[2]) - (i3 * pj[1] + i4 * pj[2]);
  T rz = i5 * pi[2] - i5 * pj[2];
  rx -= r_rint(rx); ry -= r_rint(ry); rz -= r_rint(rz);
  d[0] = B[0] * rx + B[1] * ry + B[2] * rz;
  d[1] = B[3] * ry + B[4] * rz;
  d[2] = B[5] * rz;
}

__device__ __forceinline__ int species_shift(const int* tipos, const int* actual_type) {
  int at = actual_type[0], s = 0;
  for (int y = 0; y < at; y++) s += tipos[y];
  return s;
}

// ---- radial operators that sum over neighbours.  One warp per atom: the neighbours grouped by species in shared
// memory, one lane per (species, channel) walking its group, so that no sum crosses lanes.
//   val[k]: descriptor of the k-th grouped neighbour; src[k]: its position in the row; off[q]: first of species q
struct RadStage {
  int* src;
  int* off;  // [nt + 1]
};
__device__ __forceinline__ void rad_group(const RadStage& st, const int* __restrict__ row, int n, int nt,
                                          const int* __restrict__ type_map, int lane) {
  const unsigned lt = (1u << lane) - 1u;
  int o = 0;
  for (int q = 0; q < nt; q++) {
    if (lane == 0) st.off[q] = o;
    for (int k0 = 0; k0 < n; k0 += 32) {
      const int k = k0 + lane;
      const bool p = k < n && type_map[row[k]] == q;
      const unsigned bal = __ballot_sync(0xffffffffu, p);
      if (p) st.src[o + __popc(bal & lt)] = k;
      o += __popc(bal);
    }
  }
  if (lane == 0) st.off[nt] = o;
  __syncwarp();
}
// bytes of shared memory per warp: two value rows, the source row, the offsets, a row per (species, channel)
template <class T>
static inline size_t rad_warp_bytes(int nr, int nt, int Fr) {
  return ((size_t)sizeof(T) * (2 * nr + nt * Fr) + sizeof(int) * (nr + nt + 1) + 15) & ~(size_t)15;
}
template <class T>
__device__ __forceinline__ void exp_table_load(T* et) {
  if (sizeof(T) == 8 && threadIdx.x < 16) et[threadIdx.x] = (T)EXP16_TABLE[threadIdx.x];
  if (sizeof(T) == 8) __syncthreads();
}

// MODE 0: fingerprints (ComputeSortProj); 1: their parameter gradient (ComputeTwoBodyParGrad); 2: backward of the
// radial force (ComputeForceRadialGrad).
template <class T>
struct RadArgs {
  int natoms, Nl, N, nr, Fr, nt;
  const T *rad, *alpha2b, *e2;
  const int *im2, *type_map;
  T* out;             // 0: two_body_afs; 2: gradnet
  const T* prevgrad;  // 1: [natoms, Fr]; 2: force cotangent [nf, 3N]
  T *g_alpha, *g_emb;
  const T *netderiv, *der2b;
  const int *tipos, *actual_type;
};
template <class T, int MODE>
__global__ void __launch_bounds__(OPS_THREADS) k_rad_sums(RadArgs<T> a, size_t warp_bytes, VirArgs<T> va) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T et[16];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nr = a.nr, Fr = a.Fr, nt = a.nt, nqc = nt * Fr;
  T* val = reinterpret_cast<T*>(smem_raw + w * warp_bytes);  // [nr] descriptor
  T* qv = val + nr;                                          // [nr] 2: projected force cotangent
  T* rs = qv + nr;                                           // [nt*Fr]
  RadStage st;
  st.src = reinterpret_cast<int*>(rs + nqc);
  st.off = st.src + nr;
  exp_table_load(et);
  chain_wait();
  // a warp keeps the parameter sums of its lanes over all of its atoms and adds them to the gradient once
  for (int L0 = 0; L0 < nqc; L0 += 32) {
    const int L = L0 + lane, q = L < nqc ? L / Fr : 0, c = L < nqc ? L - q * Fr : 0;
    const T al = L < nqc ? a.alpha2b[L] : T(0), ch = L < nqc ? a.e2[L] : T(0);
    T ga = T(0), ge = T(0);
    for (int gi = blockIdx.x * OPS_WARPS + w; gi < a.natoms; gi += gridDim.x * OPS_WARPS) {
      const size_t base = gi;
      const int* row = a.im2 + base * (nr + 1) + 1;
      int n = a.im2[base * (nr + 1)];
      if (n > nr) n = nr;
      rad_group(st, row, n, nt, a.type_map, lane);
      const int ng = st.off[nt];
      int b = 0, ipar = 0;
      T pix = T(0), piy = T(0), piz = T(0);
      if (MODE == 2) {
        b = gi / a.Nl;
        ipar = gi - b * a.Nl + species_shift(a.tipos, a.actual_type);
        const T* p = a.prevgrad + ((size_t)b * a.N + ipar) * 3;
        pix = p[0]; piy = p[1]; piz = p[2];
      }
      for (int g = lane; g < ng; g += 32) {
        const int k = st.src[g];
        val[g] = a.rad[base * nr + k];
        if (MODE == 2) {
          // q = sum_a (Fbar_j - Fbar_i)_a * 0.5 * dd/dr_{i,a}
          const int nj = row[k];
          const T* pj = a.prevgrad + ((size_t)b * a.N + nj) * 3;
          T wd[3] = {T(0), T(0), T(0)};
          if (va.wbar) {  // the virial cotangent shifts the neighbour's force cotangent by -(Wbar r) (grad_force/rad/reforce.cu.cc:165-234)
            T r[3];
            mic_cart(va.pos + ((size_t)b * a.N + ipar) * 3, va.pos + ((size_t)b * a.N + nj) * 3, va.box + (size_t)b * 6, r);
            const T* Wg = va.wbar + (size_t)b * 9;
#pragma unroll
            for (int x = 0; x < 3; x++) wd[x] = Wg[x * 3] * r[0] + Wg[x * 3 + 1] * r[1] + Wg[x * 3 + 2] * r[2];
          }
          const T* d2 = a.der2b + base * 3 * nr + k;
          qv[g] = T(0.5) * ((pj[0] - pix - wd[0]) * d2[0] + (pj[1] - piy - wd[1]) * d2[nr] + (pj[2] - piz - wd[2]) * d2[2 * nr]);
        }
      }
      __syncwarp();
      if (L < nqc) {
        T s0 = T(0), s1 = T(0), s2 = T(0);
        for (int g = st.off[q]; g < st.off[q + 1]; g++) {
          const T d = val[g], x = op_exp(al * d, et);
          if (MODE == 0) s0 += d * (x * ch);
          if (MODE == 1) {
            s1 += d * d * (x * ch);
            s2 += d * x;
          }
          if (MODE == 2) {
            const T qq = qv[g], sds = x * (T(1.) + al * d);
            s0 += qq * ch * sds;
            s1 += qq * (ch * x * d * (T(2.) + al * d));
            s2 += qq * sds;
          }
        }
        if (MODE != 1) rs[L] = s0;
        if (MODE != 0) {
          const T f = MODE == 1 ? a.prevgrad[base * Fr + c] : a.netderiv[base * Fr + c];
          ga += f * s1;
          ge += f * s2;
        }
      }
      __syncwarp();
      if (MODE != 1 && L0 + 32 >= nqc) {  // every (species, channel) of this atom has been formed
        for (int cc = lane; cc < Fr; cc += 32) {
          T v = T(0);
          for (int x = 0; x < nt; x++) v += rs[x * Fr + cc];
          a.out[base * Fr + cc] = v;
        }
        __syncwarp();
      }
    }
    if (MODE != 0 && L < nqc) {
      if (ga != T(0)) atomicAdd(a.g_alpha + L, ga);
      if (ge != T(0)) atomicAdd(a.g_emb + L, ge);
    }
  }
}

// ---- angular operators: staging
template <class T>
struct AngArgs {
  int Nl, N, nr, na, Fa, nt, ncls, chunk;  // chunk: channels per pass, <= ANG_CH
  const T *ang, *ds3, *alpha3b, *e3;
  const int *im2, *type_map, *numtriplet;
  T* out;              // fingerprints / forces / gradnet
  const T* prevgrad;   // gradient of the fingerprints: [.,Fa]; backward of the forces: force cotangent [nf,3N]
  T* g_alpha3;
  T* zero;             // written with zeros (the operator's third output), zero_n elements
  int zero_n;
  const T *netderiv, *der3bsupp, *der3b;
  const int *tipos, *actual_type;
};
// shared memory: T4 par[ncls][chunk] | T2 tab[nt][chunk][nr] | T ds[nr] | T acc[Fa] | T red[C][warps][32] | extra |
// int pos[nr] | int sp[nr] | int off[nt+1] | int nact[ncls] | ushort act[ncls][Fa]
template <class T>
struct AngSmem {
  int par, tab, ds, acc, red, extra, pos, sp, off, nact, act, total;
};
template <class T>
static inline AngSmem<T> ang_smem(int nr, int nt, int ncls, int Fa, int chunk, int nval, int extra) {
  AngSmem<T> L;
  int o = 0;
  auto take = [&](int bytes) { int r = o; o += (bytes + 15) & ~15; return r; };
  const int es = (int)sizeof(T);
  L.par = take(ncls * chunk * 4 * es);
  L.tab = take(nt * chunk * nr * 2 * es);
  L.ds = take(nr * es);
  L.acc = take(Fa * es);
  L.red = take(nval ? nt * (nt + 1) / 2 * ANG_WARPS * nval * es : 0);
  L.extra = take(extra * es);
  L.pos = take(nr * 4);
  L.sp = take(nr * 4);
  L.off = take((nt + 1) * 4);
  L.nact = take(ncls * 4);
  L.act = take(ncls * Fa * 2);
  L.total = o;
  return L;
}

template <class T>
struct AngStage {
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
  int m, Tn;
  T4* par;
  T2* tab;
  T *ds, *acc, *red, *extra;
  int *pos, *sp, *off, *nact;
  unsigned short* act;
  const T* et;
  __device__ __forceinline__ void carve(unsigned char* p, const AngSmem<T>& L) {
    par = reinterpret_cast<T4*>(p + L.par);
    tab = reinterpret_cast<T2*>(p + L.tab);
    ds = reinterpret_cast<T*>(p + L.ds);
    acc = reinterpret_cast<T*>(p + L.acc);
    red = reinterpret_cast<T*>(p + L.red);
    extra = reinterpret_cast<T*>(p + L.extra);
    pos = reinterpret_cast<int*>(p + L.pos);
    sp = reinterpret_cast<int*>(p + L.sp);
    off = reinterpret_cast<int*>(p + L.off);
    nact = reinterpret_cast<int*>(p + L.nact);
    act = reinterpret_cast<unsigned short*>(p + L.act);
  }
  // Warp 0 groups the angular neighbours by species (pos[g]: sorted position of the g-th grouped one, sp[g] its
  // species); the other warps list the channels of every class whose squared embedding is not zero.
  __device__ __forceinline__ void init(const AngArgs<T>& a, size_t base) {
    m = a.numtriplet[base];
    if (m > a.nr) m = a.nr;
    const long long Tl = (long long)m * (m - 1) / 2;
    Tn = Tl < a.na ? (int)Tl : a.na;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    if (w == 0) {
      const int* row = a.im2 + base * (a.nr + 1) + 1;
      for (int k = lane; k < m; k += 32) {
        sp[k] = a.type_map[row[k]];  // by position for now
        ds[k] = a.ds3[base * a.nr + k];
      }
      __syncwarp();
      int o = 0;
      for (int q = 0; q < a.nt; q++) {
        if (lane == 0) off[q] = o;
        for (int k0 = 0; k0 < m; k0 += 32) {
          const int k = k0 + lane;
          const bool p = k < m && sp[k] == q;
          const unsigned bal = __ballot_sync(0xffffffffu, p);
          if (p) pos[o + __popc(bal & lt)] = k;
          o += __popc(bal);
        }
      }
      if (lane == 0) off[a.nt] = o;
    } else {
      for (int s = w - 1; s < a.ncls; s += ANG_WARPS - 1) {
        int n = 0;
        for (int c0 = 0; c0 < a.Fa; c0 += 32) {
          const int c = c0 + lane;
          const bool p = c < a.Fa && a.e3[(size_t)s * a.Fa + c] != T(0);
          const unsigned bal = __ballot_sync(0xffffffffu, p);
          if (p) act[s * a.Fa + n + __popc(bal & lt)] = (unsigned short)c;
          n += __popc(bal);
        }
        if (lane == 0) nact[s] = n;
      }
    }
    for (int c = threadIdx.x; c < a.Fa; c += ANG_THREADS) acc[c] = T(0);
    __syncthreads();
    for (int q = 0; q < a.nt; q++)  // species by group from now on
      for (int g = off[q] + threadIdx.x; g < off[q + 1]; g += ANG_THREADS) sp[g] = q;
  }
  __device__ __forceinline__ int most_channels(const AngArgs<T>& a) const {
    int n = 0;
    for (int s = 0; s < a.ncls; s++) n = max(n, nact[s]);
    return n;
  }
  // channels of class s in the pass that starts at channel p0
  __device__ __forceinline__ int channels(const AngArgs<T>& a, int s, int p0) const {
    return max(0, min(a.chunk, nact[s] - p0));
  }
  // parameters and tables of a pass; block barriers on both sides
  __device__ __forceinline__ void tables(const AngArgs<T>& a, int p0) {
    __syncthreads();
    for (int q = threadIdx.x; q < a.ncls * a.chunk; q += ANG_THREADS) {
      const int s = q / a.chunk, i = q - s * a.chunk;
      T4 v;
      v.x = v.y = v.z = v.w = T(0);
      if (p0 + i < nact[s]) {
        const int c = act[s * a.Fa + p0 + i];
        const T* al = a.alpha3b + ((size_t)s * a.Fa + c) * 3;
        v.x = al[0]; v.y = al[1]; v.z = al[2]; v.w = a.e3[(size_t)s * a.Fa + c];
      }
      par[q] = v;
    }
    __syncthreads();
    const int ng = off[a.nt];
    for (int q = threadIdx.x; q < a.nt * a.chunk * ng; q += ANG_THREADS) {
      const int g = q % ng, qc = q / ng, i = qc % a.chunk, tq = qc / a.chunk, s = sp[g] + tq;
      if (s < a.ncls && p0 + i < nact[s]) {
        const T4 v = par[s * a.chunk + i];
        const T d = ds[pos[g]];
        T2 e;
        e.x = op_exp(v.x * d, et);
        e.y = op_exp(v.y * d, et);
        tab[qc * a.nr + g] = e;
      }
    }
    __syncthreads();
  }
  // slot of the triplet of sorted positions j < k
  __device__ __forceinline__ int slot(int j, int k) const { return (j * (2 * m - j - 1)) / 2 + k - j - 1; }
};

// The p-th pair of class (ta, tb): grouped indices ga (species ta), gb (species tb).
template <class T>
__device__ __forceinline__ void class_pair(const AngStage<T>& st, int ta, int tb, int p, int& ga, int& gb) {
  const int oa = st.off[ta], na_ = st.off[ta + 1] - oa, ob = st.off[tb], nb_ = st.off[tb + 1] - ob;
  if (ta == tb) {
    unrank_pair(p, na_, ga, gb);
    ga += oa; gb += oa;
  } else {
    const int r = p / nb_;
    ga = oa + r; gb = ob + p - r * nb_;
  }
}
template <class T>
__device__ __forceinline__ int class_pairs(const AngStage<T>& st, int ta, int tb) {
  const int na_ = st.off[ta + 1] - st.off[ta], nb_ = st.off[tb + 1] - st.off[tb];
  return ta == tb ? na_ * (na_ - 1) / 2 : na_ * nb_;
}

// Sums of NV values per thread over the block, left in red[warp][NV] for sum_warps() behind the next barrier.
template <class T, int NV>
__device__ __forceinline__ void leave_sums(T (&v)[NV], T* red) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  constexpr int SH = NV == 32 ? 0 : (NV == 16 ? 1 : 2);  // log2(32 / NV)
  const T tot = multi_reduce<T, NV>(v, lane);
  if ((lane & ((1 << SH) - 1)) == 0) red[w * NV + (lane >> SH)] = tot;
}
template <class T, int NV>
__device__ __forceinline__ T sum_warps(const T* red, int i) {
  T s = T(0);
#pragma unroll
  for (int w = 0; w < ANG_WARPS; w++) s += red[w * NV + i];
  return s;
}

// MODE 0: fingerprints (ComputeSortProj3body); 1: their parameter gradient (ComputeSortProj3bodyGrad); 2: backward of
// the angular force (ComputeForceTriplGrad).  Per triplet the force cotangent of 2 enters only through three scalars,
//   Q  = sum_a (Fb_j-Fb_i)_a dt/d(ij)_a + (Fb_k-Fb_i)_a dt/d(ik)_a,
//   Pj = sum_a (Fb_j-Fb_i)_a dfc_j,a,   Pk = sum_a (Fb_k-Fb_i)_a dfc_k,a,
// and with Z1 = e^{bt} exp(a1 sj + a2 sk), Z2 with j, k exchanged, g = 1 + bt, H1 = g Q/2 + (t/2)(a1 Pj + a2 Pk), H2
// with Pj, Pk exchanged, the channel's gradnet term is Z1 H1 + Z2 H2 and the parameter terms are its derivatives.
template <class T, int MODE>
__global__ void __launch_bounds__(ANG_THREADS) k_ang_sums(AngArgs<T> a, AngSmem<T> L, VirArgs<T> va) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T et[16];
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
  constexpr int PER = MODE == 0 ? 1 : (MODE == 1 ? 3 : 4), NV = MODE == 0 ? 8 : 32;
  AngStage<T> st;
  st.carve(smem_raw, L);
  st.et = et;
  exp_table_load(et);
  // 1, 2: directly behind the zero fill of their outputs, so everything they read is at least two kernels old
  if (MODE == 0) chain_wait();
  const size_t base = blockIdx.x;
  st.init(a, base);
  T* dF = st.extra;           // 2: [nr][3] Fbar_k - Fbar_i
  T* pn = st.extra + 3 * a.nr;  //    [nr] their projections on dfc
  if (MODE == 2) {
    const int b = (int)(base / a.Nl), ipar = (int)(base - (size_t)b * a.Nl) + species_shift(a.tipos, a.actual_type);
    const T* pgb = a.prevgrad + (size_t)b * a.N * 3;
    for (int k = threadIdx.x; k < st.m; k += ANG_THREADS) {
      const int id = a.im2[base * (a.nr + 1) + 1 + k];
      T wd[3] = {T(0), T(0), T(0)}, p = T(0);
      if (va.wbar) {  // grad_force/ang/reforce.cu.cc:274-446
        T r[3];
        mic_cart(va.pos + ((size_t)b * a.N + ipar) * 3, va.pos + ((size_t)b * a.N + id) * 3, va.box + (size_t)b * 6, r);
        const T* Wg = va.wbar + (size_t)b * 9;
#pragma unroll
        for (int x = 0; x < 3; x++) wd[x] = Wg[x * 3] * r[0] + Wg[x * 3 + 1] * r[1] + Wg[x * 3 + 2] * r[2];
      }
#pragma unroll
      for (int x = 0; x < 3; x++) {
        const T d = pgb[(size_t)id * 3 + x] - pgb[(size_t)ipar * 3 + x] - wd[x];
        dF[k * 3 + x] = d;
        p += d * a.der3bsupp[(base * 3 + x) * a.nr + k];
      }
      pn[k] = p;
    }
  }
  const T* t_row = a.ang + base * a.na;
  const T2* d3 = MODE == 2 ? reinterpret_cast<const T2*>(a.der3b) + base * 3 * a.na : nullptr;
  const int most = st.most_channels(a);
  for (int p0 = 0; p0 < most; p0 += a.chunk) {
    st.tables(a, p0);
    int ci = 0;
    for (int ta = 0; ta < a.nt; ta++) {
      for (int tb = ta; tb < a.nt; tb++, ci++) {
        const int s = ta + tb;
        if (s >= a.ncls) continue;
        const int nch = st.channels(a, s, p0), np = class_pairs(st, ta, tb);
        T v[NV];
#pragma unroll
        for (int x = 0; x < NV; x++) v[x] = T(0);
        const T4* par = st.par + s * a.chunk;
        const T2* tA = st.tab + (size_t)tb * a.chunk * a.nr;  // entries of the ta neighbours for partners of species tb
        const T2* tB = st.tab + (size_t)ta * a.chunk * a.nr;
        if (nch > 0)
          for (int p = threadIdx.x; p < np; p += ANG_THREADS) {
            int ga, gb;
            class_pair(st, ta, tb, p, ga, gb);
            const int ka = st.pos[ga], kb = st.pos[gb];
            const int nn = st.slot(min(ka, kb), max(ka, kb));
            if (nn >= st.Tn) continue;
            const T t = t_row[nn], sa = st.ds[ka], sb = st.ds[kb];
            T Qh = T(0), Pa = T(0), Pb = T(0);
            if (MODE == 2) {
              const int j = min(ka, kb), k = max(ka, kb);
#pragma unroll
              for (int x = 0; x < 3; x++) {
                const T2 id = d3[(size_t)x * a.na + nn];
                Qh += dF[j * 3 + x] * id.x + dF[k * 3 + x] * id.y;
              }
              Qh *= T(0.5);
              Pa = T(0.5) * t * pn[ka];
              Pb = T(0.5) * t * pn[kb];
            }
#pragma unroll
            for (int c = 0; c < ANG_CH; c++) {
              if (c >= nch) break;
              const T4 pr = par[c];
              const T2 A = tA[c * a.nr + ga], B = tB[c * a.nr + gb];
              const T E = op_exp(pr.z * t, et);
              const T Z1 = E * (A.x * B.y), Z2 = E * (A.y * B.x);
              if (MODE == 0) v[c] += t * (Z1 + Z2);
              if (MODE == 1) {
                v[4 * c] += t * (Z1 * sa + Z2 * sb);
                v[4 * c + 1] += t * (Z1 * sb + Z2 * sa);
                v[4 * c + 2] += t * t * (Z1 + Z2);
              }
              if (MODE == 2) {
                const T gQ = (T(1) + pr.z * t) * Qh;
                const T H1 = gQ + pr.x * Pa + pr.y * Pb, H2 = gQ + pr.x * Pb + pr.y * Pa;
                v[4 * c] += Z1 * H1 + Z2 * H2;
                v[4 * c + 1] += Z1 * (sa * H1 + Pa) + Z2 * (sb * H2 + Pb);
                v[4 * c + 2] += Z1 * (sb * H1 + Pb) + Z2 * (sa * H2 + Pa);
                v[4 * c + 3] += t * (Z1 * (H1 + Qh) + Z2 * (H2 + Qh));
              }
            }
          }
        leave_sums<T, NV>(v, st.red + ci * ANG_WARPS * NV);
      }
    }
    if (MODE != 0) chain_wait();
    __syncthreads();
    // totals: fingerprints and gradnet per channel in acc (a channel may belong to several classes), parameter
    // gradients to global memory, one add per block
    ci = 0;
    for (int ta = 0; ta < a.nt; ta++) {
      for (int tb = ta; tb < a.nt; tb++, ci++) {
        const int s = ta + tb;
        if (s >= a.ncls) continue;
        const int nch = st.channels(a, s, p0);
        const T* red = st.red + ci * ANG_WARPS * NV;
        for (int x = threadIdx.x; x < nch * PER; x += ANG_THREADS) {
          const int i = x / PER, k = x - i * PER, c = st.act[s * a.Fa + p0 + i];
          const T f = T(0.5) * st.par[s * a.chunk + i].w * sum_warps<T, NV>(red, MODE == 0 ? i : 4 * i + k);
          if (MODE == 0 || (MODE == 2 && k == 0)) st.acc[c] += f;  // one thread per channel of the class
          else {
            const T g = f * (MODE == 1 ? a.prevgrad[base * a.Fa + c] : a.netderiv[base * a.Fa + c]);
            atomicAdd(a.g_alpha3 + ((size_t)s * a.Fa + c) * 3 + (MODE == 1 ? k : k - 1), g);
          }
        }
        __syncthreads();
      }
    }
  }
  if (MODE != 0) chain_wait();
  if (MODE != 1) {
    __syncthreads();
    for (int c = threadIdx.x; c < a.Fa; c += ANG_THREADS) a.out[base * a.Fa + c] = st.acc[c];
  }
  if (MODE != 0 && base == 0)
    for (int c = threadIdx.x; c < a.zero_n; c += ANG_THREADS) a.zero[c] = T(0);
}

// ---------------------------------------------------------------- radial force (ComputeForceRadial)
template <class T>
__global__ void __launch_bounds__(OPS_THREADS)
    k_force_rad(int natoms, int Nl, int N, int nr, int Fr, const T* __restrict__ netderiv,
                const T* __restrict__ der2b, const int* __restrict__ im2, const T* __restrict__ rad,
                const T* __restrict__ alpha2b, const T* __restrict__ e2, const int* __restrict__ type_map,
                const int* __restrict__ tipos, const int* __restrict__ actual_type, T* __restrict__ force,
                VirArgs<T> va) {
  const int gi = blockIdx.x * OPS_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (gi >= natoms) return;
  chain_wait();
  const int b = gi / Nl, par = gi - b * Nl;
  const int ipar = par + species_shift(tipos, actual_type);
  const size_t base = gi;
  int n = im2[base * (nr + 1)];
  if (n > nr) n = nr;
  T fx = T(0), fy = T(0), fz = T(0);
  T vw[9];
#pragma unroll
  for (int c = 0; c < 9; c++) vw[c] = T(0);
  for (int j = lane; j < n; j += 32) {
    const int nj = im2[base * (nr + 1) + 1 + j];
    const int tj = type_map[nj];
    const T d = rad[base * nr + j];
    T w = T(0);
    for (int c = 0; c < Fr; c++) {
      const T ch = e2[Fr * tj + c];
      if (ch == T(0)) continue;
      const T al = alpha2b[Fr * tj + c];
      T sds = ch * r_exp(al * d);
      sds *= (T(1.) + al * d);
      w += netderiv[base * Fr + c] * (T(0.5) * sds);
    }
    const T gx = w * der2b[(base * 3 + 0) * nr + j];
    const T gy = w * der2b[(base * 3 + 1) * nr + j];
    const T gz = w * der2b[(base * 3 + 2) * nr + j];
    T* fj = force + ((size_t)b * N + nj) * 3;
    atomicAdd(fj + 0, gx);
    atomicAdd(fj + 1, gy);
    atomicAdd(fj + 2, gz);
    fx -= gx; fy -= gy; fz -= gz;
    if (va.virial) {  // W_ab -= g_a r_b (force/rad/reforce.cu.cc:174-287)
      T r[3];
      mic_cart(va.pos + ((size_t)b * N + ipar) * 3, va.pos + ((size_t)b * N + nj) * 3, va.box + (size_t)b * 6, r);
      const T g[3] = {gx, gy, gz};
#pragma unroll
      for (int a = 0; a < 3; a++)
#pragma unroll
        for (int c = 0; c < 3; c++) vw[a * 3 + c] -= g[a] * r[c];
    }
  }
  fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz);
  if (lane == 0) {
    T* fi = force + ((size_t)b * N + ipar) * 3;
    atomicAdd(fi + 0, fx);
    atomicAdd(fi + 1, fy);
    atomicAdd(fi + 2, fz);
  }
  if (va.virial) {
#pragma unroll
    for (int c = 0; c < 9; c++) {
      const T v = warp_sum(vw[c]);
      if (lane == 0) atomicAdd(va.virial + (size_t)b * 9 + c, v);
    }
  }
}

// ---------------------------------------------------------------- angular force (ComputeForceTripl)
// Ordered pairs: four threads share a neighbour and walk its partners, so that the force on it stays in registers
// until the end; every triplet is evaluated from both sides (one exponential per channel each).
constexpr int ANG_TPO = 4;
template <class T>
__global__ void __launch_bounds__(ANG_THREADS) k_force_ang(AngArgs<T> a, AngSmem<T> L, VirArgs<T> va) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T et[16];
  __shared__ T red[ANG_WARPS + 1];
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
  AngStage<T> st;
  st.carve(smem_raw, L);
  st.et = et;
  exp_table_load(et);
  const size_t base = blockIdx.x;
  const int b = (int)(base / a.Nl), par_ = (int)(base - (size_t)b * a.Nl);
  const int ipar = par_ + species_shift(a.tipos, a.actual_type);
  st.init(a, base);
  T* fnb = st.extra;  // [nr][3] force on the neighbour at sorted position k
  for (int q = threadIdx.x; q < 3 * a.nr; q += ANG_THREADS) fnb[q] = T(0);
  const T* t_row = a.ang + base * a.na;
  const T2* d3 = reinterpret_cast<const T2*>(a.der3b) + base * 3 * a.na;
  const int most = st.most_channels(a), ng = st.off[a.nt], sub = threadIdx.x & (ANG_TPO - 1);
  for (int p0 = 0; p0 < most; p0 += a.chunk) {
    st.tables(a, p0);
    for (int g0 = 0; g0 < ng; g0 += ANG_THREADS / ANG_TPO) {
      const int g = g0 + threadIdx.x / ANG_TPO;
      T f[3] = {T(0), T(0), T(0)};
      if (g < ng) {
        const int kj = st.pos[g], tj = st.sp[g];
        T sup = T(0);
        for (int tq = 0; tq < a.nt; tq++) {
          const int s = tj + tq;
          if (s >= a.ncls) continue;
          const int nch = st.channels(a, s, p0);
          if (nch <= 0) continue;
          const T4* par = st.par + s * a.chunk;
          const T2* tA = st.tab + (size_t)tq * a.chunk * a.nr + g;
          const T2* tB = st.tab + (size_t)tj * a.chunk * a.nr;
          T w[ANG_CH];
          T2 A[ANG_CH];
#pragma unroll
          for (int c = 0; c < ANG_CH; c++) {
            w[c] = T(0);
            A[c].x = A[c].y = T(0);
            if (c < nch) {
              w[c] = T(0.25) * a.netderiv[base * a.Fa + st.act[s * a.Fa + p0 + c]] * par[c].w;
              A[c] = tA[c * a.nr];
              A[c].x *= w[c]; A[c].y *= w[c];
            }
          }
          for (int h = st.off[tq] + sub; h < st.off[tq + 1]; h += ANG_TPO) {
            if (h == g) continue;
            const int kk = st.pos[h];
            const int nn = st.slot(min(kj, kk), max(kj, kk));
            if (nn >= st.Tn) continue;
            const T t = t_row[nn];
            T D = T(0), B = T(0);
#pragma unroll
            for (int c = 0; c < ANG_CH; c++) {
              if (c >= nch) break;
              const T4 pr = par[c];
              const T2 P = tB[c * a.nr + h];
              const T E = op_exp(pr.z * t, et);
              const T Z1 = E * (A[c].x * P.y), Z2 = E * (A[c].y * P.x);
              D += (T(1) + pr.z * t) * (Z1 + Z2);
              B += pr.x * Z1 + pr.y * Z2;
            }
            sup += B * t;
            const bool first = kj < kk;
#pragma unroll
            for (int x = 0; x < 3; x++) {
              const T2 id = d3[(size_t)x * a.na + nn];
              f[x] += D * (first ? id.x : id.y);
            }
          }
        }
#pragma unroll
        for (int x = 0; x < 3; x++) f[x] += sup * a.der3bsupp[(base * 3 + x) * a.nr + kj];
      }
#pragma unroll
      for (int x = 0; x < 3; x++) {
        f[x] += __shfl_xor_sync(0xffffffffu, f[x], 1);
        f[x] += __shfl_xor_sync(0xffffffffu, f[x], 2);
      }
      if (g < ng && sub < 3) fnb[st.pos[g] * 3 + sub] += sub == 0 ? f[0] : (sub == 1 ? f[1] : f[2]);
    }
  }
  __syncthreads();
  chain_wait();
  T* fb = a.out + (size_t)b * a.N * 3;
  const int* row = a.im2 + base * (a.nr + 1) + 1;
  T fi[3] = {T(0), T(0), T(0)};
  for (int k = threadIdx.x; k < st.m; k += ANG_THREADS) {
#pragma unroll
    for (int x = 0; x < 3; x++) fi[x] -= fnb[k * 3 + x];
  }
  for (int q = threadIdx.x; q < st.m * 3; q += ANG_THREADS) atomicAdd(fb + (size_t)row[q / 3] * 3 + (q % 3), fnb[q]);
#pragma unroll
  for (int x = 0; x < 3; x++) {
    const T v = block_sum<T, ANG_WARPS>(fi[x], red);
    if (threadIdx.x == 0) atomicAdd(fb + (size_t)ipar * 3 + x, v);
  }
  if (va.virial && threadIdx.x < 32) {
    // W_ab -= f_ij,a r_ij,b + f_ik,a r_ik,b (force/ang/reforce.cu.cc:269-457): every force this centre puts on
    // neighbour k multiplies the same r_ik, so the per-neighbour totals suffice
    T w[9];
#pragma unroll
    for (int c = 0; c < 9; c++) w[c] = T(0);
    for (int k = threadIdx.x; k < st.m; k += 32) {
      T r[3];
      mic_cart(va.pos + ((size_t)b * a.N + ipar) * 3, va.pos + ((size_t)b * a.N + row[k]) * 3, va.box + (size_t)b * 6, r);
#pragma unroll
      for (int x = 0; x < 3; x++)
#pragma unroll
        for (int c = 0; c < 3; c++) w[x * 3 + c] -= fnb[k * 3 + x] * r[c];
    }
#pragma unroll
    for (int c = 0; c < 9; c++) {
      const T v = warp_sum(w[c]);
      if (threadIdx.x == 0) atomicAdd(va.virial + (size_t)b * 9 + c, v);
    }
  }
}

// ================================================================= launchers
template <class T>
static int ops_check(stafb_ctx* c) {
  if (!c) return STAFB_ERR_INVALID;
  if ((c->dtype == STAFB_F32) != (sizeof(T) == 4)) return STAFB_ERR_INVALID;
  return STAFB_OK;
}

// Dynamic shared memory above 48 KB has to be asked for, per kernel and device.
static cudaError_t opt_in(const void* kern, size_t bytes) {
  return bytes > 48 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)
                           : cudaSuccess;
}

static inline int ncls_of(int nt) {
  int C = nt * (nt + 1) / 2, smax = 2 * nt - 1;
  return C < smax ? C : smax;
}

// k_rad_sums on `n` atoms: at most eight warps' worth of blocks per SM, so that a warp's parameter sums cover several
// atoms of a large batch before they meet the other warps' in global memory.
template <class T, int MODE>
static int launch_rad(cudaStream_t s, const RadArgs<T>& a, VirArgs<T> va = VirArgs<T>()) {
  const size_t wb = rad_warp_bytes<T>(a.nr, a.nt, a.Fr), sm = wb * OPS_WARPS;
  STAFB_CUDA_OK(opt_in((const void*)k_rad_sums<T, MODE>, sm));
  const int blocks = (a.natoms + OPS_WARPS - 1) / OPS_WARPS, cap = MODE == 0 ? blocks : 148 * 8;
  STAFB_CUDA_OK(launch_chained(k_rad_sums<T, MODE>, blocks < cap ? blocks : cap, OPS_THREADS, sm, s, a, wb, va));
  return STAFB_OK;
}

// Shared memory of an angular operator: as many channels per pass as fit, ANG_CH if possible.
template <class T>
static int ang_layout(AngArgs<T>& a, int nval, int extra, AngSmem<T>& L) {
  for (a.chunk = ANG_CH; a.chunk >= 1; a.chunk >>= 1) {
    L = ang_smem<T>(a.nr, a.nt, a.ncls, a.Fa, a.chunk, nval, extra);
    if (L.total <= 200 * 1024) return STAFB_OK;
  }
  return STAFB_ERR_CAPACITY;
}
template <class T, int MODE>
static int launch_ang(cudaStream_t s, int blocks, AngArgs<T> a, VirArgs<T> va = VirArgs<T>()) {
  AngSmem<T> L;
  const int rc = ang_layout<T>(a, MODE == 0 ? 8 : 32, MODE == 2 ? 4 * a.nr : 0, L);
  if (rc != STAFB_OK) return rc;
  STAFB_CUDA_OK(opt_in((const void*)k_ang_sums<T, MODE>, (size_t)L.total));
  STAFB_CUDA_OK(launch_chained(k_ang_sums<T, MODE>, blocks, ANG_THREADS, (size_t)L.total, s, a, L, va));
  return STAFB_OK;
}
template <class T>
static AngArgs<T> ang_args(stafb_ctx* c, const T* ang, const T* ds3, const int* im2, const T* a3, const T* e3,
                           const int* tm, const int* ntr, int nt, int Fa) {
  AngArgs<T> a = {};
  a.nr = c->nr; a.na = c->na; a.Fa = Fa; a.nt = nt; a.ncls = ncls_of(nt);
  a.ang = ang; a.ds3 = ds3; a.im2 = im2; a.alpha3b = a3; a.e3 = e3; a.type_map = tm; a.numtriplet = ntr;
  return a;
}
template <class T>
static RadArgs<T> rad_args(stafb_ctx* c, const T* rad, const int* im2, const T* a2, const T* e2, const int* tm, int n,
                           int nt, int Fr) {
  RadArgs<T> a = {};
  a.natoms = n; a.nr = c->nr; a.Fr = Fr; a.nt = nt;
  a.rad = rad; a.im2 = im2; a.alpha2b = a2; a.e2 = e2; a.type_map = tm;
  return a;
}

template <class T>
int op_sort_proj(stafb_ctx* c, cudaStream_t s, const T* rad, const int* im2, const T* a2, const T* e2,
                 const int* tm, int nf, int Nl, int nt, int Fr, T* out) {
  const int n = nf * Nl;
  if (n <= 0) return STAFB_OK;
  RadArgs<T> a = rad_args<T>(c, rad, im2, a2, e2, tm, n, nt, Fr);
  a.out = out;
  return launch_rad<T, 0>(s, a);
}

template <class T>
int op_sort_proj3(stafb_ctx* c, cudaStream_t s, const T* ang, const T* ds3, const int* im2, const T* a3, const T* e3,
                  const int* tm, const int* ntr, int nf, int Nl, int nt, int Fa, T* out) {
  const int n = nf * Nl;
  if (n <= 0) return STAFB_OK;
  AngArgs<T> a = ang_args<T>(c, ang, ds3, im2, a3, e3, tm, ntr, nt, Fa);
  a.out = out;
  return launch_ang<T, 0>(s, n, a);
}

template <class T>
int op_force_rad(stafb_ctx* c, cudaStream_t s, const T* nd, const T* der2b, const int* im2, const T* rad,
                 const T* a2, const T* e2, const int* tm, const int* tipos, const int* at, int nf, int Nl, int N,
                 int nt, int Fr, T* force, VirArgs<T> va = VirArgs<T>()) {
  STAFB_CUDA_OK(zero_two(s, force, sizeof(T) * (size_t)nf * 3 * N, va.virial, va.virial ? sizeof(T) * (size_t)nf * 9 : 0));
  const int n = nf * Nl;
  if (n <= 0) return STAFB_OK;
  STAFB_CUDA_OK(launch_chained(k_force_rad<T>, (n + OPS_WARPS - 1) / OPS_WARPS, OPS_THREADS, 0, s, n, Nl, N, c->nr, Fr,
                               nd, der2b, im2, rad, a2, e2, tm, tipos, at, force, va));
  return STAFB_OK;
}

template <class T>
int op_force_ang(stafb_ctx* c, cudaStream_t s, const T* nd, const T* ds3, const T* ang, const T* d3s, const T* d3,
                 const int* im2, const T* a3, const T* e3, const int* tm, const int* tipos, const int* at,
                 const int* ntr, int nf, int Nl, int N, int nt, int Fa, T* force, VirArgs<T> va = VirArgs<T>()) {
  STAFB_CUDA_OK(zero_two(s, force, sizeof(T) * (size_t)nf * 3 * N, va.virial, va.virial ? sizeof(T) * (size_t)nf * 9 : 0));
  const int n = nf * Nl;
  if (n <= 0) return STAFB_OK;
  AngArgs<T> a = ang_args<T>(c, ang, ds3, im2, a3, e3, tm, ntr, nt, Fa);
  a.Nl = Nl; a.N = N; a.netderiv = nd; a.der3bsupp = d3s; a.der3b = d3; a.tipos = tipos; a.actual_type = at; a.out = force;
  AngSmem<T> L;
  const int rc = ang_layout<T>(a, 0, 3 * a.nr, L);
  if (rc != STAFB_OK) return rc;
  STAFB_CUDA_OK(opt_in((const void*)k_force_ang<T>, (size_t)L.total));
  STAFB_CUDA_OK(launch_chained(k_force_ang<T>, n, ANG_THREADS, (size_t)L.total, s, a, L, va));
  return STAFB_OK;
}

template <class T>
int op_grad_af_rad(stafb_ctx* c, cudaStream_t s, const T* pg, const T* rad, const int* im2, const T* a2, const T* e2,
                   const int* tm, int nf, int Nl, int nt, int Fr, T* ga, T* ge) {
  if (nt > STAFB_MAX_TYPES) return STAFB_ERR_INVALID;
  STAFB_CUDA_OK(zero_two(s, ga, sizeof(T) * nt * Fr, ge, sizeof(T) * nt * Fr));
  const int n = nf * Nl;
  if (n <= 0) return STAFB_OK;
  RadArgs<T> a = rad_args<T>(c, rad, im2, a2, e2, tm, n, nt, Fr);
  a.prevgrad = pg; a.g_alpha = ga; a.g_emb = ge;
  return launch_rad<T, 1>(s, a);
}

template <class T>
int op_grad_af_ang(stafb_ctx* c, cudaStream_t s, const T* pg, const T* ang, const T* ds3, const int* im2,
                   const T* a3, const T* e3, const int* tm, const int* ntr, int nf, int Nl, int nt, int Fa, T* ga,
                   T* ge) {
  const int C = nt * (nt + 1) / 2, n = nf * Nl;
  STAFB_CUDA_OK(zero_two(s, ga, sizeof(T) * C * 3 * Fa, ge, n > 0 ? 0 : sizeof(T) * C * Fa));
  if (n <= 0) return STAFB_OK;
  AngArgs<T> a = ang_args<T>(c, ang, ds3, im2, a3, e3, tm, ntr, nt, Fa);
  a.prevgrad = pg; a.g_alpha3 = ga; a.zero = ge; a.zero_n = C * Fa;
  return launch_ang<T, 1>(s, n, a);
}

template <class T>
int op_grad_force_rad(stafb_ctx* c, cudaStream_t s, const T* pg, const T* nd, const T* der2b, const int* im2,
                      const T* rad, const T* a2, const T* e2, const int* tm, const int* tipos, const int* at, int nf,
                      int Nl, int N, int nt, int Fr, T* gradnet, T* ga, T* ge, VirArgs<T> va = VirArgs<T>()) {
  if (nt > STAFB_MAX_TYPES) return STAFB_ERR_INVALID;
  STAFB_CUDA_OK(zero_two(s, ga, sizeof(T) * nt * Fr, ge, sizeof(T) * nt * Fr));
  const int n = nf * Nl;
  if (n <= 0) return STAFB_OK;
  RadArgs<T> a = rad_args<T>(c, rad, im2, a2, e2, tm, n, nt, Fr);
  a.Nl = Nl; a.N = N; a.prevgrad = pg; a.netderiv = nd; a.der2b = der2b; a.tipos = tipos; a.actual_type = at;
  a.out = gradnet; a.g_alpha = ga; a.g_emb = ge;
  return launch_rad<T, 2>(s, a, va);
}

template <class T>
int op_grad_force_ang(stafb_ctx* c, cudaStream_t s, const T* pg, const T* nd, const T* ds3, const T* ang,
                      const T* d3s, const T* d3, const int* im2, const T* a3, const T* e3, const int* tm,
                      const int* tipos, const int* at, const int* ntr, int nf, int Nl, int N, int nt, int Fa,
                      T* gradnet, T* ga, T* gck, VirArgs<T> va = VirArgs<T>()) {
  const int C = nt * (nt + 1) / 2, n = nf * Nl;
  STAFB_CUDA_OK(zero_two(s, ga, sizeof(T) * C * 3 * Fa, gck, n > 0 ? 0 : sizeof(T) * C * Fa));
  if (n <= 0) return STAFB_OK;
  AngArgs<T> a = ang_args<T>(c, ang, ds3, im2, a3, e3, tm, ntr, nt, Fa);
  a.Nl = Nl; a.N = N; a.prevgrad = pg; a.netderiv = nd; a.der3bsupp = d3s; a.der3b = d3; a.tipos = tipos;
  a.actual_type = at; a.out = gradnet; a.g_alpha3 = ga; a.zero = gck; a.zero_n = C * Fa;
  return launch_ang<T, 2>(s, n, a, va);
}

}  // namespace stafb

using namespace stafb;
#define DISPATCH(c, call_f, call_d)                               \
  do {                                                            \
    if (!(c)) return STAFB_ERR_INVALID;                           \
    cudaStream_t s = (cudaStream_t)stream;                        \
    if ((c)->dtype == STAFB_F32) { typedef float R; return call_f; } \
    typedef double R;                                             \
    return call_d;                                                \
  } while (0)

extern "C" int stafb_compute_sort_proj(stafb_ctx* c, void* stream, const void* rad, const int* im2, const void* a2,
                                       const void* e2, const int* tm, int nf, int Nl, int nt, int Fr, void* out) {
  DISPATCH(c, op_sort_proj<R>(c, s, (const R*)rad, im2, (const R*)a2, (const R*)e2, tm, nf, Nl, nt, Fr, (R*)out),
           op_sort_proj<R>(c, s, (const R*)rad, im2, (const R*)a2, (const R*)e2, tm, nf, Nl, nt, Fr, (R*)out));
}

extern "C" int stafb_compute_sort_proj3body(stafb_ctx* c, void* stream, const void* ang, const void* ds3,
                                            const int* im3, const int* im2, const void* a3, const void* e3,
                                            const int* tm, const int* ntr, int nf, int Nl, int nt, int Fa,
                                            void* out) {
  (void)im3;  // the pair ids are recomputed from interaction_map_rad; same values by construction
  DISPATCH(c,
           op_sort_proj3<R>(c, s, (const R*)ang, (const R*)ds3, im2, (const R*)a3, (const R*)e3, tm, ntr, nf, Nl, nt,
                            Fa, (R*)out),
           op_sort_proj3<R>(c, s, (const R*)ang, (const R*)ds3, im2, (const R*)a3, (const R*)e3, tm, ntr, nf, Nl, nt,
                            Fa, (R*)out));
}

extern "C" int stafb_compute_force_radial(stafb_ctx* c, void* stream, const void* nd, const void* der2b,
                                          const int* im2, const void* rad, const void* a2, const void* e2,
                                          const int* tm, const int* tipos, const int* at, int nf, int Nl, int N,
                                          int nt, int Fr, void* force) {
  DISPATCH(c,
           op_force_rad<R>(c, s, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2, (const R*)e2, tm,
                           tipos, at, nf, Nl, N, nt, Fr, (R*)force),
           op_force_rad<R>(c, s, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2, (const R*)e2, tm,
                           tipos, at, nf, Nl, N, nt, Fr, (R*)force));
}

extern "C" int stafb_compute_force_tripl(stafb_ctx* c, void* stream, const void* nd, const void* ds3, const void* ang,
                                         const void* d3s, const void* d3, const int* im2, const int* im3,
                                         const void* a3, const void* e3, const int* tm, const int* tipos,
                                         const int* at, const int* ntr, int nf, int Nl, int N, int nt, int Fa,
                                         void* force) {
  (void)im3;
  DISPATCH(c,
           op_force_ang<R>(c, s, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s, (const R*)d3, im2,
                           (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa, (R*)force),
           op_force_ang<R>(c, s, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s, (const R*)d3, im2,
                           (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa, (R*)force));
}

extern "C" int stafb_compute_two_body_par_grad(stafb_ctx* c, void* stream, const void* pg, const void* rad,
                                               const int* im2, const void* a2, const void* e2, const int* tm, int nf,
                                               int Nl, int nt, int Fr, void* ga, void* ge) {
  DISPATCH(c,
           op_grad_af_rad<R>(c, s, (const R*)pg, (const R*)rad, im2, (const R*)a2, (const R*)e2, tm, nf, Nl, nt, Fr,
                             (R*)ga, (R*)ge),
           op_grad_af_rad<R>(c, s, (const R*)pg, (const R*)rad, im2, (const R*)a2, (const R*)e2, tm, nf, Nl, nt, Fr,
                             (R*)ga, (R*)ge));
}

extern "C" int stafb_compute_sort_proj3body_grad(stafb_ctx* c, void* stream, const void* pg, const void* ang,
                                                 const void* ds3, const int* im3, const int* im2, const void* a3,
                                                 const void* e3, const int* tm, const int* ntr, int nf, int Nl,
                                                 int nt, int Fa, void* ga, void* ge) {
  (void)im3;
  DISPATCH(c,
           op_grad_af_ang<R>(c, s, (const R*)pg, (const R*)ang, (const R*)ds3, im2, (const R*)a3, (const R*)e3, tm,
                             ntr, nf, Nl, nt, Fa, (R*)ga, (R*)ge),
           op_grad_af_ang<R>(c, s, (const R*)pg, (const R*)ang, (const R*)ds3, im2, (const R*)a3, (const R*)e3, tm,
                             ntr, nf, Nl, nt, Fa, (R*)ga, (R*)ge));
}

extern "C" int stafb_compute_force_radial_grad(stafb_ctx* c, void* stream, const void* pg, const void* nd,
                                               const void* der2b, const int* im2, const void* rad, const void* a2,
                                               const void* e2, const int* tm, const int* tipos, const int* at,
                                               int nf, int Nl, int N, int nt, int Fr, void* gradnet, void* ga,
                                               void* ge) {
  DISPATCH(c,
           op_grad_force_rad<R>(c, s, (const R*)pg, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2,
                                (const R*)e2, tm, tipos, at, nf, Nl, N, nt, Fr, (R*)gradnet, (R*)ga, (R*)ge),
           op_grad_force_rad<R>(c, s, (const R*)pg, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2,
                                (const R*)e2, tm, tipos, at, nf, Nl, N, nt, Fr, (R*)gradnet, (R*)ga, (R*)ge));
}

extern "C" int stafb_compute_force_tripl_grad(stafb_ctx* c, void* stream, const void* pg, const void* nd,
                                              const void* ds3, const void* ang, const void* d3s, const void* d3,
                                              const int* im2, const int* im3, const void* a3, const void* e3,
                                              const int* tm, const int* tipos, const int* at, const int* ntr, int nf,
                                              int Nl, int N, int nt, int Fa, void* gradnet, void* ga, void* gck) {
  (void)im3;
  DISPATCH(c,
           op_grad_force_ang<R>(c, s, (const R*)pg, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s,
                                (const R*)d3, im2, (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa,
                                (R*)gradnet, (R*)ga, (R*)gck),
           op_grad_force_ang<R>(c, s, (const R*)pg, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s,
                                (const R*)d3, im2, (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa,
                                (R*)gradnet, (R*)ga, (R*)gck));
}


// ---- ...Virial / ...VirialGrad variants: the same kernels with the positions, the box and the virial (or its
// cotangent) attached
template <class R>
static VirArgs<R> vir_args(const void* pos, const void* box, void* virial, const void* wbar) {
  VirArgs<R> va;
  va.pos = (const R*)pos; va.box = (const R*)box; va.virial = (R*)virial; va.wbar = (const R*)wbar;
  return va;
}

extern "C" int stafb_compute_force_radial_virial(stafb_ctx* c, void* stream, const void* nd, const void* der2b,
                                                 const int* im2, const void* rad, const void* a2, const void* e2,
                                                 const int* tm, const int* tipos, const int* at, const void* pos,
                                                 const void* box, int nf, int Nl, int N, int nt, int Fr, void* force,
                                                 void* virial) {
  if (!pos || !box || !virial) return STAFB_ERR_INVALID;
  DISPATCH(c,
           op_force_rad<R>(c, s, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2, (const R*)e2, tm,
                           tipos, at, nf, Nl, N, nt, Fr, (R*)force, vir_args<R>(pos, box, virial, nullptr)),
           op_force_rad<R>(c, s, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2, (const R*)e2, tm,
                           tipos, at, nf, Nl, N, nt, Fr, (R*)force, vir_args<R>(pos, box, virial, nullptr)));
}

extern "C" int stafb_compute_force_tripl_virial(stafb_ctx* c, void* stream, const void* nd, const void* ds3,
                                                const void* ang, const void* d3s, const void* d3, const int* im2,
                                                const int* im3, const void* a3, const void* e3, const int* tm,
                                                const int* tipos, const int* at, const int* ntr, const void* pos,
                                                const void* box, int nf, int Nl, int N, int nt, int Fa, void* force,
                                                void* virial) {
  (void)im3;
  if (!pos || !box || !virial) return STAFB_ERR_INVALID;
  DISPATCH(c,
           op_force_ang<R>(c, s, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s, (const R*)d3, im2,
                           (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa, (R*)force,
                           vir_args<R>(pos, box, virial, nullptr)),
           op_force_ang<R>(c, s, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s, (const R*)d3, im2,
                           (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa, (R*)force,
                           vir_args<R>(pos, box, virial, nullptr)));
}

extern "C" int stafb_compute_force_radial_virial_grad(stafb_ctx* c, void* stream, const void* pg, const void* pgv,
                                                      const void* nd, const void* der2b, const int* im2,
                                                      const void* rad, const void* a2, const void* e2, const int* tm,
                                                      const int* tipos, const int* at, const void* pos,
                                                      const void* box, int nf, int Nl, int N, int nt, int Fr,
                                                      void* gradnet, void* ga, void* ge) {
  if (!pos || !box || !pgv) return STAFB_ERR_INVALID;
  DISPATCH(c,
           op_grad_force_rad<R>(c, s, (const R*)pg, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2,
                                (const R*)e2, tm, tipos, at, nf, Nl, N, nt, Fr, (R*)gradnet, (R*)ga, (R*)ge,
                                vir_args<R>(pos, box, nullptr, pgv)),
           op_grad_force_rad<R>(c, s, (const R*)pg, (const R*)nd, (const R*)der2b, im2, (const R*)rad, (const R*)a2,
                                (const R*)e2, tm, tipos, at, nf, Nl, N, nt, Fr, (R*)gradnet, (R*)ga, (R*)ge,
                                vir_args<R>(pos, box, nullptr, pgv)));
}

extern "C" int stafb_compute_force_tripl_virial_grad(stafb_ctx* c, void* stream, const void* pg, const void* pgv,
                                                     const void* nd, const void* ds3, const void* ang,
                                                     const void* d3s, const void* d3, const int* im2, const int* im3,
                                                     const void* a3, const void* e3, const int* tm, const int* tipos,
                                                     const int* at, const int* ntr, const void* pos, const void* box,
                                                     int nf, int Nl, int N, int nt, int Fa, void* gradnet, void* ga,
                                                     void* gck) {
  (void)im3;
  if (!pos || !box || !pgv) return STAFB_ERR_INVALID;
  DISPATCH(c,
           op_grad_force_ang<R>(c, s, (const R*)pg, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s,
                                (const R*)d3, im2, (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa,
                                (R*)gradnet, (R*)ga, (R*)gck, vir_args<R>(pos, box, nullptr, pgv)),
           op_grad_force_ang<R>(c, s, (const R*)pg, (const R*)nd, (const R*)ds3, (const R*)ang, (const R*)d3s,
                                (const R*)d3, im2, (const R*)a3, (const R*)e3, tm, tipos, at, ntr, nf, Nl, N, nt, Fa,
                                (R*)gradnet, (R*)ga, (R*)gck, vir_args<R>(pos, box, nullptr, pgv)));
}
