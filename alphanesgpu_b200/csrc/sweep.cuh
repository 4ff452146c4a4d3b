// Sweep kernels of the fused path (included by model.cuh inside namespace stafb): atomic fingerprints, forces and
// the backward of the forces, each as one pass over the triplets of every central atom.
//
// One warp owns one central atom.  Its neighbour record (common.cuh: unit vectors, cutoffs, radial descriptors,
// neighbour ids, grouped by species) and the per-species parameter block that k_prep packs once per evaluation
// arrive in shared memory by two bulk asynchronous copies that complete on an mbarrier; nothing about the
// geometry is recomputed here except the angle of a pair.
//
// Triplets are enumerated per species-pair class (ta <= tb) rather than in the reference's j<k slot order: inside
// a class every triplet uses the same parameter row (row = type_j + type_k,
// STAF/src/fingerprint/ang/reforce.cu.cc:56), so the channel loop is uniform across the warp and channels whose
// squared embedding is zero are skipped for the whole class.  exp(a1*sj + a2*sk) is formed as a product of
// per-neighbour factors exp(a1*sj), exp(a2*sk) tabulated once per (class, channel chunk); in fp32 all
// exponentials are base-2 (one MUFU.EX2) with parameters pre-scaled by log2(e), two channels per packed
// instruction.  The force sweep walks ORDERED pairs so that every lane accumulates the force on "its" neighbour
// in registers; the other sweeps walk unordered pairs and reduce per-lane sums with a transposing butterfly.
//
// Math: STAF/src/fingerprint, force, grad_finger, grad_force (rad and ang) reforce.cu.cc and
// STAF/staf_models/staf_model.py:168-258 of the reference (see include/stafb.h).
#pragma once

constexpr int MAXP = 4;  // channel PAIRS processed per pass over the pairs of a class
constexpr int FP_CH = 5;  // channels per pass of the partner-packed fp32 force sweep: 4 FP_CH owner constants in registers
constexpr int FP_REC = FP_CH + 2;  // 16-byte words of a partner pair's record (odd)
// Exponential tables: entry (neighbour k, channel pair lp) at tab4[k * TSTR + lp].  Neighbour-major, so that the
// entries of one neighbour are at constant offsets from one address; the odd stride (5 x 16 bytes) keeps the
// 16-byte loads of lanes on consecutive neighbours free of bank conflicts.
constexpr int TSTR = MAXP + 1;

// ---- bulk asynchronous copy global -> shared, completion on an mbarrier (this GPU's own memory only)
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned arrivals) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(arrivals) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// dst, src 16-byte aligned; bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Bounded wait for a phase of the barrier; false if the copies did not land (the caller records a status and
// leaves, it never spins for ever).
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
  for (int it = 0; it < (1 << 24); it++) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// 2^x for a pre-scaled argument: one MUFU.EX2 (results below 2^-126 flush to zero; arguments here are products
// of exponents of magnitude <= ~10 with cutoff values in [0,1], far from overflow)
__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// exponential of a pre-scaled argument; et: the 16-entry table in shared memory (double only)
template <class T> struct Ex;
template <> struct Ex<float> {
  static __host__ __device__ __forceinline__ float scale() { return 1.4426950408889634f; }
  static __device__ __forceinline__ float f(float x, const float*) { return ex2_fast(x); }
};
template <> struct Ex<double> {
  static __host__ __device__ __forceinline__ double scale() { return 1.0; }
  static __device__ __forceinline__ double f(double x, const double* et) { return exp_table16(x, et); }
};

// Two-channel packed arithmetic.  On sm_100 a float2 multiply / add / fma is ONE instruction (__fmul2_rn,
// __fadd2_rn, __ffma2_rn), so the channel loops carry two channels per instruction; double pairs are two scalar
// operations.  `one`: only the first channel of the pair exists (double; an odd channel count would otherwise cost
// the exponentials of a channel that contributes nothing - in fp32 the padding channel rides along in the packed
// instruction).  It is a compile-time constant once the channel loops are unrolled.
__device__ __forceinline__ float2 p_mul(float2 a, float2 b, bool = false) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 p_add(float2 a, float2 b, bool = false) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 p_fma(float2 a, float2 b, float2 c, bool = false) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ double2 p_mul(double2 a, double2 b, bool one = false) {
  return make_double2(a.x * b.x, one ? 0.0 : a.y * b.y);
}
__device__ __forceinline__ double2 p_add(double2 a, double2 b, bool one = false) {
  return make_double2(a.x + b.x, one ? 0.0 : a.y + b.y);
}
__device__ __forceinline__ double2 p_fma(double2 a, double2 b, double2 c, bool one = false) {
  return make_double2(a.x * b.x + c.x, one ? c.y : a.y * b.y + c.y);
}
__device__ __forceinline__ float2 mk2(float x, float y) { return make_float2(x, y); }
__device__ __forceinline__ double2 mk2(double x, double y) { return make_double2(x, y); }
__device__ __forceinline__ float2 p_ex(float2 a, const float* et, bool = false) {
  return make_float2(Ex<float>::f(a.x, et), Ex<float>::f(a.y, et));
}
__device__ __forceinline__ double2 p_ex(double2 a, const double* et, bool one = false) {
  return make_double2(Ex<double>::f(a.x, et), one ? 0.0 : Ex<double>::f(a.y, et));
}

// AFV = fingerprints that also leave d(AF)/d(alpha) per atom (training)
enum { MODE_AF = 0, MODE_FORCE = 1, MODE_FGRAD = 2, MODE_AFV = 4 };

// Resident one-warp blocks per SM the kernels are compiled for (caps the registers per thread at
// 65536 / (32 * blocks)); the hardware holds at most 32 blocks per SM.
// fp32: 96 registers, five warps per scheduler = 20 blocks per SM (the shared memory of a block allows the same).  A
// batch of 4 x 768 atoms is 20.8 blocks per SM; the few that do not fit start as the first ones retire.  Capping at
// 80 registers for 24 blocks was measured: spills, and no gain in the chained step.
template <int MODE, size_t ES> struct SweepMinBlocks { static constexpr int value = 20; };
template <> struct SweepMinBlocks<MODE_AF, 8> { static constexpr int value = 16; };          // <= 128
template <> struct SweepMinBlocks<MODE_AFV, 8> { static constexpr int value = 12; };         // <= 168
template <> struct SweepMinBlocks<MODE_FORCE, 8> { static constexpr int value = 8; };        // no spills at <= 255
template <> struct SweepMinBlocks<MODE_FGRAD, 8> { static constexpr int value = 8; };        // <= 255

// ---- per-species parameter block (global memory, written by k_prep at the start of every evaluation; a sweep
// copies the block of its central species into shared memory).  Byte offsets inside a block:
//   [0, 32)  int nact[8]            active channels (squared embedding != 0) of class s = ta + tb
//   [32, 48) int nrad[4]            active radial channels of neighbour species q
//   actc     uchar [ncls][Famax]    their channel numbers, compacted
//   chq      T4 [ncls][maxp]        channel pair (2p, 2p+1) of the compacted list: alpha1 x2, alpha2 x2
//   chr      T2 [ncls][maxp]        beta x2
//   che      T2 [ncls][maxp]        squared embedding x2 (an odd count is padded with an all-zero channel)
//   rpar     T4 [nt][Frmax]         active radial channels, compacted: alpha2b*log2(e), alpha2b, squared embedding, channel
//                                   number; the rest of a row is zero
struct SparLayout {
  int actc, chq, chr, che, rpar, total, maxp;
};
template <class T>
static inline SparLayout spar_layout(const ModelDev& d) {
  SparLayout L;
  int o = 48;
  auto take = [&](int bytes) { int r = o; o += (bytes + 15) & ~15; return r; };
  L.maxp = (d.Famax + 1) / 2 > 0 ? (d.Famax + 1) / 2 : 1;
  L.actc = take(d.ncls * (d.Famax > 0 ? d.Famax : 1));
  L.chq = take(d.ncls * L.maxp * 4 * (int)sizeof(T));
  L.chr = take(d.ncls * L.maxp * 2 * (int)sizeof(T));
  L.che = take(d.ncls * L.maxp * 2 * (int)sizeof(T));
  L.rpar = take(d.nt * (d.Frmax > 0 ? d.Frmax : 1) * 4 * (int)sizeof(T));
  L.total = o;
  return L;
}

// What the rounding of alpha * log2(e) to fp32 drops: alike for every atom, it would not average out of the gradient.
template <class T>
__device__ __forceinline__ T scale_rest(T al, T als) {
  if constexpr (sizeof(T) == 8) return T(0);
  else return fmaf(al, 1.442695022f, -als) + al * 1.925963e-8f;
}

// Fills the block of (species t, class s): one warp; lanes over channels, ballot compaction of the active ones.
template <class T>
__device__ __forceinline__ void spar_fill_class(const ModelDev& md, const SparLayout& sl, unsigned char* blk, int t,
                                                int s, const T* __restrict__ theta, const T* __restrict__ emb,
                                                int lane) {
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
  const int Fa = md.Fa[t], Fr = md.Fr[t], nt = md.nt;
  const T* a3 = theta + md.off_a3[t] + (size_t)s * 3 * Fa;
  const T* e3 = emb + md.off_emb[t] + nt * Fr + (size_t)s * Fa;
  unsigned char* actc = blk + sl.actc + s * md.Famax;
  T* chq = reinterpret_cast<T*>(blk + sl.chq) + (size_t)s * sl.maxp * 4;
  T* chr = reinterpret_cast<T*>(blk + sl.chr) + (size_t)s * sl.maxp * 2;
  T* che = reinterpret_cast<T*>(blk + sl.che) + (size_t)s * sl.maxp * 2;
  const unsigned lt = (1u << lane) - 1u;
  int nact = 0;
  for (int c0 = 0; c0 < Fa; c0 += 32) {
    const int c = c0 + lane;
    const T ee = c < Fa ? e3[c] : T(0);
    // fetched beside the embedding, not after it
    const T al1 = c < Fa ? a3[3 * c] : T(0), al2 = c < Fa ? a3[3 * c + 1] : T(0), be = c < Fa ? a3[3 * c + 2] : T(0);
    const bool p = ee != T(0);
    const unsigned bal = __ballot_sync(0xffffffffu, p);
    if (p) {
      const int slot = nact + __popc(bal & lt), pr = slot >> 1, h = slot & 1;
      actc[slot] = (unsigned char)c;
      chq[pr * 4 + h] = al1; chq[pr * 4 + 2 + h] = al2;
      chr[pr * 2 + h] = be;
      che[pr * 2 + h] = ee;
    }
    nact += __popc(bal);
  }
  if (lane == 0) {
    reinterpret_cast<int*>(blk)[s] = nact;
    if (nact & 1) {  // the partner of the last channel: a channel that contributes nothing
      const int pr = nact >> 1;
      chq[pr * 4 + 1] = T(0); chq[pr * 4 + 3] = T(0);
      chr[pr * 2 + 1] = T(0);
      che[pr * 2 + 1] = T(0);
    }
  }
}

// The radial channels of (species t, neighbour species q): one warp, as above.
template <class T>
__device__ __forceinline__ void spar_fill_radial(const ModelDev& md, const SparLayout& sl, unsigned char* blk, int t, int q,
                                                 const T* __restrict__ theta, const T* __restrict__ emb, int lane) {
  const int Fr = md.Fr[t];
  T* row = reinterpret_cast<T*>(blk + sl.rpar) + (size_t)q * md.Frmax * 4;
  int nact = 0;
  for (int c0 = 0; c0 < Fr; c0 += 32) {
    const int c = c0 + lane;
    const T ee = c < Fr ? emb[md.off_emb[t] + q * Fr + c] : T(0);
    const T al = c < Fr ? theta[md.off_a2[t] + q * Fr + c] : T(0);
    const bool p = ee != T(0);
    const unsigned bal = __ballot_sync(0xffffffffu, p);
    if (p) {
      T* rp = row + (nact + __popc(bal & ((1u << lane) - 1u))) * 4;
      rp[0] = al * Ex<T>::scale(); rp[1] = al; rp[2] = ee; rp[3] = (T)c;
    }
    nact += __popc(bal);
  }
  for (int x = 4 * nact + lane; x < 4 * md.Frmax; x += 32) row[x] = T(0);
  if (lane == 0) reinterpret_cast<int*>(blk)[8 + q] = nact;
}

// The virial of a frame is accumulated by every centre of the frame: 9 words would take one atomic add per atom
// each (24,576 on one address for a large box), so every component has VIR_SLOTS words, a centre adds to slot
// (its index mod VIR_SLOTS) and the readers sum the slots.  Layout [frame][9][VIR_SLOTS] doubles.
constexpr int VIR_SLOTS = 32;
__device__ __forceinline__ double vir_total(const double* __restrict__ vacc, int frame, int q) {
  const double* p = vacc + ((size_t)frame * 9 + q) * VIR_SLOTS;
  double w = 0.0;
#pragma unroll 8
  for (int s = 0; s < VIR_SLOTS; s++) w += p[s];
  return w;
}

template <class T>
struct SweepArgs {
  const unsigned char* rows;  // [nf, N] neighbour records
  int row_stride;             // bytes
  int nr, nf, nall;           // nall: atoms per frame in the force / cotangent arrays (>= N: ghosts)
  const unsigned char* spar;  // [nt] parameter blocks
  int spar_stride;
  SparLayout sl;
  const T* chan_in;  // FORCE/FGRAD: netderiv[nf,N,Fmax]
  const T* force;    // FGRAD: forces [nf,3*nall] and their labels; dL/dF = fscale * L'(force - label) with L the
  const T* flab;     //        Huber (loss_kind 0) or the squared error
  T fscale;
  int loss_kind;
  T* out;            // AF/AFV: af[nf,N,Fmax]; FORCE: force[nf,3*nall]; FGRAD: gradnet[nf,N,Fmax]
  T* grad;           // FGRAD: flat parameter gradient (accumulated)
  T* vout;           // AFV: d(AF)/d(alpha) rows [nf,N,nv] in the accumulator layout (alpha2b[nt,Frmax] | alpha3b[C,3*Famax])
  int nv;
  double* vir;       // FORCE with VIR: virial accumulators [nf,9,VIR_SLOTS]
  const double* vacc;  // FGRAD with a virial loss: the accumulators the force sweep filled, the labels [nf,9] and
  const T* vlab;       //        the loss's scale: dL/dW = vscale * L'(W - label)
  T vscale;
  int* status;
};

// partner pairs of the fp32 force sweep at most
__host__ __device__ inline int fp_pairs(int nr) { return (nr + STAFB_MAX_TYPES + 1) / 2; }

// shared-memory layout of a sweep block (byte offsets)
struct SweepSmem {
  int row, spar, tab, xtra, part, acc, rsum, wch, red, etab, mbar, total;
};
template <class T>
static inline SweepSmem sweep_smem(const ModelDev& d, const SparLayout& sl, int nr, int mode, int nw, bool pack) {
  SweepSmem L;
  int o = 0;
  auto take = [&](int bytes) { int r = o; o += (bytes + 15) & ~15; return r; };
  const int es = (int)sizeof(T);
  L.row = take(row_stride_bytes(nr, es));
  L.spar = take(sl.total);
  // PACK: the records of the partner pairs (every species group padded to a pair), channel weights and beta of a pass
  L.tab = take(pack ? FP_REC * fp_pairs(nr) * 16 + FP_CH * 24 : TSTR * nr * 4 * es);
  L.xtra = take(mode == MODE_FORCE ? 3 * nr * es : (mode == MODE_FGRAD ? 4 * nr * es : 0));
  L.part = take(mode == MODE_FORCE && nw > 1 ? 3 * 32 * nw * es : 0);  // forces of the segments of an owner
  L.acc = take(mode == MODE_FORCE ? 0 : (d.nt * d.Frmax + d.C * 3 * d.Famax + d.Famax) * es);
  L.rsum = take(d.nt * (d.Frmax > 0 ? d.Frmax : 1) * es);
  L.wch = take(mode == MODE_FORCE ? d.ncls * sl.maxp * 2 * es : 0);
  L.red = take(32 * es);  // group offsets
  L.etab = take(es == 8 ? 16 * es : 0);  // table of the double exponential
  L.mbar = take(16);
  L.total = o;
  return L;
}

// Barrier over the NW warps of a block, and an addition into shared memory that only one lane per warp makes.
template <int NW>
__device__ __forceinline__ void block_sync() {
  if (NW == 1) __syncwarp(); else __syncthreads();
}
template <int NW, class T>
__device__ __forceinline__ void acc_add(T* p, T v) {
  if (NW == 1) *p += v; else atomicAdd(p, v);
}

// Pairs of a class as a rectangle of rows x cols walked LANES positions at a time without divisions.  Two different
// species (SAME == false): rows = neighbours of ta, cols = neighbours of tb.  One species with n neighbours: the
// strict upper triangle j < k folded into a rectangle - row r of the triangle (n-1-r entries) is followed by row
// n-1-r (n even) or n-2-r (n odd), which together have n-1 (n) entries.
template <bool SAME, int LANES>
struct PairWalk {
  int r, c, cols, qs, rs, nm1, odd;
  __device__ __forceinline__ void init(int na, int nb, int lane) {
    odd = na & 1;
    nm1 = na - 1;
    cols = SAME ? (odd ? na : na - 1) : nb;
    if (cols < 1) cols = 1;
    r = lane / cols;
    c = lane - r * cols;
    qs = LANES / cols;
    rs = LANES - qs * cols;
  }
  __device__ __forceinline__ static int count(int na, int nb) { return SAME ? na * (na - 1) / 2 : na * nb; }
  __device__ __forceinline__ void get(int& j, int& k) const {
    if (SAME) {
      const bool first = c < nm1 - r;
      j = first ? r : nm1 - odd - r;
      k = first ? r + 1 + c : c + 1 - odd;
    } else {
      j = r;
      k = c;
    }
  }
  __device__ __forceinline__ void step() {
    r += qs;
    c += rs;
    if (c >= cols) { c -= cols; r++; }
  }
};

// ---- unordered pairs: fingerprints (AF), fingerprints + d(AF)/d(alpha) (AFV), backward of the forces (FGRAD).
// Per-lane sums r[v][lp] (v = 0: fingerprint / gradnet, 1..3: alpha1, alpha2, beta terms) for NCHP channel pairs.
template <class T, int MODE, int NCH, bool SAME, int NW, int NCHP = (NCH + 1) / 2>
__device__ __forceinline__ void pairs_unordered(const typename Vec4<T>::type* __restrict__ U,
                                                const typename Vec4<T>::type* __restrict__ V,
                                                const typename Vec4<T>::type* __restrict__ dF,
                                                const typename Vec4<T>::type* __restrict__ tab4, int nr,
                                                const typename Vec4<T>::type* __restrict__ chq,
                                                const typename Vec2<T>::type* __restrict__ chr, const T* __restrict__ et,
                                                int oa, int ob,
                                                int na_, int nb_, int lane,
                                                typename Vec2<T>::type (&r0)[NCHP], typename Vec2<T>::type (&r1)[NCHP],
                                                typename Vec2<T>::type (&r2)[NCHP],
                                                typename Vec2<T>::type (&r3)[NCHP]) {
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
#pragma unroll
  for (int lp = 0; lp < NCHP; lp++) r0[lp] = r1[lp] = r2[lp] = r3[lp] = mk2(T(0), T(0));
  const T2 one2 = mk2(T(1), T(1));
  constexpr bool ODD = sizeof(T) == 8 && (NCH & 1);
  const int np = PairWalk<SAME, 32 * NW>::count(na_, nb_);
  PairWalk<SAME, 32 * NW> pw;
  pw.init(na_, nb_, lane);
  // beta of every channel pair stays in registers in the fingerprint modes
  T2 bsc[NCHP];
  if (MODE != MODE_FGRAD) {
#pragma unroll
    for (int lp = 0; lp < NCHP; lp++) bsc[lp] = chr[lp];
  }
  // pairs in flight per lane: two hide the shared-memory and exponential latencies of the fingerprint loops; the
  // force-backward loop is too large for that (its unrolled body falls out of the instruction cache)
  constexpr int PAIR_UNROLL = (MODE == MODE_FGRAD) ? 1 : 2;
#pragma unroll PAIR_UNROLL
  for (int p = lane; p < np; p += 32 * NW) {
    int jj, kk;
    pw.get(jj, kk);
    pw.step();
    const int j = oa + jj, k = ob + kk;
    const T4 uj = U[j], uk = U[k];
    const T fcj = uj.w, fck = uk.w;
    const T cs = uj.x * uk.x + uj.y * uk.y + uj.z * uk.z;
    const T half = T(0.5) * cs + T(0.5);
    const T tt = half * fcj * fck;
    const T ts = tt * Ex<T>::scale();  // exp(beta t) as 2^(beta ts) in fp32
    const T2 tt2 = mk2(tt, tt), ts2 = mk2(ts, ts), fcj2 = mk2(fcj, fcj), fck2 = mk2(fck, fck);
    if (MODE != MODE_FGRAD) {
#pragma unroll
      for (int lp = 0; lp < NCHP; lp++) {
        const bool h = ODD && lp == NCHP - 1;
        const T4 A = tab4[j * TSTR + lp], B = tab4[k * TSTR + lp];
        const T2 S1 = p_mul(mk2(A.z, A.w), mk2(B.x, B.y), h);  // exp(a2*sj + a1*sk)
        const T2 S2 = p_mul(mk2(A.x, A.y), mk2(B.z, B.w), h);  // exp(a1*sj + a2*sk)
        const T2 cm = p_mul(p_ex(p_mul(bsc[lp], ts2, h), et, h), tt2, h);  // t*exp(beta*t)
        const T2 ss = p_add(S1, S2, h);
        r0[lp] = p_fma(cm, ss, r0[lp], h);  // the channel coefficient is applied after the reduction
        if (MODE == MODE_AFV) {
          r1[lp] = p_fma(cm, p_fma(S2, fcj2, p_mul(S1, fck2, h), h), r1[lp], h);
          r2[lp] = p_fma(cm, p_fma(S2, fck2, p_mul(S1, fcj2, h), h), r2[lp], h);
          r3[lp] = p_fma(p_mul(cm, tt2, h), ss, r3[lp], h);
        }
      }
    } else {
      // Backward of the triplet force for the cotangent dF_k = Fbar_k - Fbar_i (dF.w = dF . u).  With
      //   Q  = d(t)/d(positions) . dF  (symmetric in j,k),  Pj = fc'_j (dF_j . u_j),  Pk likewise,
      //   Z1 = E exp(a1 sj + a2 sk), Z2 = E exp(a2 sj + a1 sk), E = exp(beta t), g = 1 + beta t,
      //   H1 = g Q/2 + (t/2)(a1 Pj + a2 Pk),  H2 = g Q/2 + (t/2)(a1 Pk + a2 Pj)
      // the channel's gradnet term is  Z1 H1 + Z2 H2  (the two orderings of the pair) and the parameter terms are
      // its derivatives:  d/da1 = Z1 (sj H1 + t Pj/2) + Z2 (sk H2 + t Pk/2),  d/da2 with sj, sk and Pj, Pk
      // exchanged inside each bracket,  d/dbeta = t [Z1 (H1 + Q/2) + Z2 (H2 + Q/2)]
      // (STAF/src/grad_force/ang/reforce.cu.cc:47-231).
      // What depends on one neighbour only is formed before the pair loop: dF[k] holds W/4 with W = fc/r (dF - (dF.u) u)
      // and q/2 with q = dfc/dr (dF.u), and
      //   Q = fc_k W_j.u_k / 2 + fc_j W_k.u_j / 2 + (1 + cos)/2 (fc_k q_j + fc_j q_k),
      // 13 operations where the pair's four products with dF, 1/r and dfc/dr took 27 (eight steps of 4 x 768 atoms in fp64
      // 2,557 -> 2,498 us, of the wide model in fp32 2,730 -> 2,676 us, with the compacted radial channels).
      const T4 Wj = dF[j], Wk = dF[k];
      const T wju = Wj.x * uk.x + Wj.y * uk.y + Wj.z * uk.z;
      const T wku = Wk.x * uj.x + Wk.y * uj.y + Wk.z * uj.z;
      const T Qh = half * (fck * Wj.w + fcj * Wk.w) + (fck * wju + fcj * wku);
      const T Pjh = tt * Wj.w, Pkh = tt * Wk.w;
      const T2 Qh2 = mk2(Qh, Qh), Pj2 = mk2(Pjh, Pjh), Pk2 = mk2(Pkh, Pkh);
#pragma unroll
      for (int lp = 0; lp < NCHP; lp++) {
        const bool h = ODD && lp == NCHP - 1;
        const T4 A = tab4[j * TSTR + lp], B = tab4[k * TSTR + lp], cq = chq[lp];
        const T2 be = chr[lp];
        const T2 al1 = mk2(cq.x, cq.y), al2 = mk2(cq.z, cq.w);
        const T2 E = p_ex(p_mul(be, ts2, h), et, h);
        const T2 Z1 = p_mul(E, p_mul(mk2(A.x, A.y), mk2(B.z, B.w), h), h);
        const T2 Z2 = p_mul(E, p_mul(mk2(A.z, A.w), mk2(B.x, B.y), h), h);
        const T2 gQ = p_mul(p_fma(be, tt2, one2, h), Qh2, h);
        const T2 H1 = p_fma(al1, Pj2, p_fma(al2, Pk2, gQ, h), h), H2 = p_fma(al1, Pk2, p_fma(al2, Pj2, gQ, h), h);
        r0[lp] = p_fma(Z1, H1, p_fma(Z2, H2, r0[lp], h), h);
        r1[lp] = p_fma(Z1, p_fma(fcj2, H1, Pj2, h), p_fma(Z2, p_fma(fck2, H2, Pk2, h), r1[lp], h), h);
        r2[lp] = p_fma(Z1, p_fma(fck2, H1, Pk2, h), p_fma(Z2, p_fma(fcj2, H2, Pj2, h), r2[lp], h), h);
        r3[lp] = p_fma(tt2, p_fma(Z1, p_add(H1, Qh2, h), p_mul(Z2, p_add(H2, Qh2, h), h), h), r3[lp], h);
      }
    }
  }
}

// Adds the forces of the segments of an owner, which lie on consecutive lanes, to the owner's: one thread per (owner,
// component).  (A shared float atomic is a compare-and-swap loop: S lanes on one word cost S round trips, most of the time
// of a force pass when four warps share an atom and S goes up to 16.)
template <class T, int NW>
__device__ __forceinline__ void flush_segments(int oo, int base, int S, int nseg, int lane, T fx, T fy, T fz,
                                               T* __restrict__ fo, T* __restrict__ part) {
  part[lane * 3] = fx; part[lane * 3 + 1] = fy; part[lane * 3 + 2] = fz;
  block_sync<NW>();
  const int o0 = base / S, last = min(nseg - base, 32 * NW), cnt = (base + last - 1) / S + 1 - o0;
  for (int q = lane; q < 3 * cnt; q += 32 * NW) {
    const int o = o0 + q / 3, c = q % 3, l1 = min((o + 1) * S - base, last);
    T f = T(0);
    for (int l = max(o * S - base, 0); l < l1; l++) f += part[l * 3 + c];
    fo[(oo + o) * 3 + c] += f;
  }
  block_sync<NW>();
}

// ---- ordered pairs (owner j, partner k): forces.  The list of an owner's partners is cut into S segments and
// every lane takes one (owner, segment): the owner's data - including its table entries already multiplied by the
// channel weights - and its force accumulator stay in registers for the whole segment, all lanes run the same
// number of iterations, and the accumulators are flushed once per round (S lanes share an owner).  S in 1..4 is
// chosen per class to fill the 32 lanes.  fo[k*3 + a]: force on neighbour k; (fix, fiy, fiz): on the centre.
template <class T, int NCH, bool SAME, int NW, int NCHP = (NCH + 1) / 2>
__device__ __forceinline__ void pairs_force(const typename Vec4<T>::type* __restrict__ U,
                                            const typename Vec4<T>::type* __restrict__ V,
                                            const typename Vec4<T>::type* __restrict__ tab4,
                                            const typename Vec4<T>::type* __restrict__ chq,
                                            const typename Vec2<T>::type* __restrict__ chr,
                                            const typename Vec2<T>::type* __restrict__ wch, const T* __restrict__ et,
                                            int oo, int op, int no, int npt, int lane, T* __restrict__ fo,
                                            T* __restrict__ part, T& fix, T& fiy, T& fiz) {
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
  if (no <= 0 || npt <= 0) return;
  // segments per owner: fewest (iterations + 2) * rounds; the 2 stands for loading the owner and flushing
  int S = 1, seg = npt, best = 0x7fffffff;
#pragma unroll
  for (int s = 1; s <= (NW == 1 ? 4 : 16); s++) {
    const int sg = (npt + s - 1) / s, rounds = (no * s + 32 * NW - 1) / (32 * NW), cost = rounds * (sg + 2);
    if (cost < best) { best = cost; S = s; seg = sg; }
  }
  constexpr int FORCE_UNROLL = sizeof(T) == 4 ? 2 : 1;  // two partners in flight where the registers allow it
  constexpr bool ODD = sizeof(T) == 8 && (NCH & 1);
  const int nseg = no * S;
  const T2 one2 = mk2(T(1), T(1));
  for (int base = 0; base < nseg; base += 32 * NW) {
    const int sidx = base + lane;
    const bool active = sidx < nseg;
    int ow = 0;  // sidx / S (the reciprocal is exact for these ranges)
    if (active) {
      if (NW == 1) ow = (S == 1) ? sidx : (S == 2) ? (sidx >> 1) : (S == 4) ? (sidx >> 2) : (sidx * 21846) >> 16;
      else ow = (sidx * ((65535 + S) / S)) >> 16;
    }
    const int k0 = (sidx - ow * S) * seg;
    const int j = oo + ow;
    const T4 uj = U[j];
    const T4 vj = V[j];
    const T rinvj = vj.x, gfcj = vj.y;
    T2 a1w[NCHP], a2w[NCHP], b1w[NCHP], b2w[NCHP];  // w*A1_j, w*A2_j, alpha1*w*A1_j, alpha2*w*A2_j
#pragma unroll
    for (int lp = 0; lp < NCHP; lp++) {
      const T4 A = tab4[j * TSTR + lp], cq = chq[lp];
      const T2 w = wch[lp];
      a1w[lp] = p_mul(mk2(A.x, A.y), w);
      a2w[lp] = p_mul(mk2(A.z, A.w), w);
      b1w[lp] = p_mul(mk2(cq.x, cq.y), a1w[lp]);
      b2w[lp] = p_mul(mk2(cq.z, cq.w), a2w[lp]);
    }
    T ax = T(0), ay = T(0), az = T(0), as = T(0);
    // this lane's partners [k0, k1); for one species the owner itself is skipped: partner kb >= ow is row kb + 1
    const int k1 = active ? ((k0 + seg < npt) ? k0 + seg : npt) : k0;
#pragma unroll FORCE_UNROLL
    for (int kb = k0; kb < k1; kb++) {
      {
        const int k = op + kb + ((SAME && kb >= ow) ? 1 : 0);
        const T4 uk = U[k];
        const T cs = uj.x * uk.x + uj.y * uk.y + uj.z * uk.z;
        const T half = T(0.5) * cs + T(0.5);
        const T tt = half * uj.w * uk.w;
        const T ts = tt * Ex<T>::scale();
        const T2 tt2 = mk2(tt, tt), ts2 = mk2(ts, ts);
        T2 D2 = mk2(T(0), T(0)), BJ2 = mk2(T(0), T(0));
#pragma unroll
        for (int lp = 0; lp < NCHP; lp++) {
          const T4 B = tab4[k * TSTR + lp];
          const T2 be = chr[lp];
          const T2 A1k = mk2(B.x, B.y), A2k = mk2(B.z, B.w);
          const bool h = ODD && lp == NCHP - 1;
          const T2 Ex2 = p_ex(p_mul(be, ts2, h), et, h);
          const T2 sum = p_fma(a1w[lp], A2k, p_mul(a2w[lp], A1k, h), h);                // w (S2 + S1)
          D2 = p_fma(p_mul(p_fma(be, tt2, one2, h), Ex2, h), sum, D2, h);  // w e^{bt} (1 + bt) (S1 + S2)
          BJ2 = p_fma(Ex2, p_fma(b1w[lp], A2k, p_mul(b2w[lp], A1k, h), h), BJ2, h);     // w e^{bt} (a1 S2 + a2 S1)
        }
        const T D = D2.x + D2.y, BJ = (BJ2.x + BJ2.y) * tt;
        // f_ij = cjk*u_k + (...)*u_j
        const T cjk = D * T(0.5) * uj.w * uk.w * rinvj;
        ax += cjk * uk.x; ay += cjk * uk.y; az += cjk * uk.z;
        as += -cs * cjk + gfcj * (D * half * uk.w + BJ);
      }
    }
    if (NW == 1) {
      if (active) {
        const T fx = ax + as * uj.x, fy = ay + as * uj.y, fz = az + as * uj.z;
        atomicAdd(&fo[j * 3 + 0], fx);
        atomicAdd(&fo[j * 3 + 1], fy);
        atomicAdd(&fo[j * 3 + 2], fz);
        fix -= fx; fiy -= fy; fiz -= fz;
      }
    } else {
      const T fx = ax + as * uj.x, fy = ay + as * uj.y, fz = az + as * uj.z;
      if (active) { fix -= fx; fiy -= fy; fiz -= fz; }
      flush_segments<T, NW>(oo, base, S, nseg, lane, fx, fy, fz, fo, part);
    }
  }
}

// ---- the same in fp32 with TWO PARTNERS per packed instruction (the PACK form of the kernel, for models with FP_CH
// channels per class or fewer: the geometry is formed once per pass of FP_CH channels, and with 13 channels the form above
// with its eight per pass is the faster one, 73 against 78 us).  Packing channels leaves the geometry of a pair, its force
// and the loop itself scalar and pads five channels to six; packing partners halves all of it.  For that the partners lie
// in pairs, one record of FP_REC 16-byte words per pair: x x' y y' | z z' fc/2 fc'/2 | per channel exp(a1 fc) of both,
// exp(a2 fc) of both.  Every species group starts a pair, an odd group ends with a partner of cutoff zero, which adds
// nothing, and within one species the owner itself is masked the same way.  Lanes with the same segment number read the
// same record (one address per load and segment; the odd record length keeps different segments out of each other's
// banks).  The owner's constants are 64-bit registers that hold the value twice, made where the compiler cannot see that
// the halves agree: left to itself it keeps one copy and spends a move per use.  Against the form above: training step of
// 4 x 768 atoms 160.3 -> 159.0 us, of 2 x 96 85.5 -> 83.9 us, 6,144-atom domain 133.0 -> 131.0 us, 24,576-atom call 541 ->
// 537 us: instruction issue is still the bound, and half of the sweep's instructions lie outside the pair loop.
typedef unsigned long long f2x;
__device__ __forceinline__ f2x x_dup(float v) {
  f2x r;
  asm volatile("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ f2x x_pack(float a, float b) {
  f2x r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 x_split(f2x v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2x x_mul(f2x a, f2x b) {
  f2x r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2x x_fma(f2x a, f2x b, f2x c) {
  f2x r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// Segments per owner of a pass: fewest (iterations + 2) * rounds; the 2 stands for loading the owner and flushing.  Lane s
// weighs s + 1 segments.
template <int NW>
__device__ __forceinline__ int choose_segments(int no, int npt) {
  constexpr int MOST = NW == 1 ? 4 : 16;
  const int s = (threadIdx.x & (MOST - 1)) + 1;
  const int sg = (npt + s - 1) / s, rounds = (no * s + 32 * NW - 1) / (32 * NW);
  return (int)(__reduce_min_sync(0xffffffffu, (unsigned)(rounds * (sg + 2) * 32 + s)) & 31u);
}
template <int NCH, bool SAME, int NW>
__device__ __forceinline__ void pairs_force2(const float4* __restrict__ U, const float4* __restrict__ V,
                                             const float4* __restrict__ rec, const f2x* __restrict__ beta,
                                             const float4* __restrict__ cw, int oo, int jp0, int kp0, int no, int npp,
                                             int lane, float* __restrict__ fo, float* __restrict__ part, float& fix,
                                             float& fiy, float& fiz) {
  if (no <= 0 || npp <= 0) return;
  const int S = choose_segments<NW>(no, npp), seg = (npp + S - 1) / S;
  const int nseg = no * S;
  const f2x one2 = x_dup(1.0f);
  for (int base = 0; base < nseg; base += 32 * NW) {
    const int sidx = base + lane;
    const bool active = sidx < nseg;
    int ow = 0;  // sidx / S (exact for these ranges)
    if (active) {
      if (NW == 1) ow = (S == 1) ? sidx : (S == 2) ? (sidx >> 1) : (S == 4) ? (sidx >> 2) : (sidx * 21846) >> 16;
      else ow = (sidx * ((65535 + S) / S)) >> 16;
    }
    const int pos = sidx - ow * S, s0 = pos * seg;
    const int j = oo + ow, jp = jp0 + (ow >> 1);
    const float4 uj = U[j];
    f2x a1w[NCH], a2w[NCH], b1w[NCH], b2w[NCH];  // w*A1_j, w*A2_j, alpha1*w*A1_j, alpha2*w*A2_j
#pragma unroll
    for (int c = 0; c < NCH; c++) {
      const float* A = reinterpret_cast<const float*>(rec + jp * FP_REC + 2 + c) + (ow & 1);
      const float4 w = cw[c];  // weight, alpha1 * weight, alpha2 * weight
      const float A1 = A[0], A2 = A[2];
      a1w[c] = x_dup(A1 * w.x);
      a2w[c] = x_dup(A2 * w.x);
      b1w[c] = x_dup(A1 * w.y);
      b2w[c] = x_dup(A2 * w.z);
    }
    const f2x ux = x_dup(uj.x), uy = x_dup(uj.y), uz = x_dup(uj.z), fj = x_dup(uj.w),
              fs = x_dup(uj.w * Ex<float>::scale());
    f2x ax = 0, ay = 0, az = 0, ac = 0, ah = 0;  // bit patterns of (0, 0)
    const int s1 = active ? min(s0 + seg, npp) : s0;
    const ulonglong2* r = reinterpret_cast<const ulonglong2*>(rec + (kp0 + s0) * FP_REC);
    const int hole = SAME ? (ow >> 1) - s0 : 0;  // the step that meets the owner itself
#pragma unroll 1
    for (int p = 0; p < s1 - s0; p++, r += FP_REC) {
      const ulonglong2 g0 = r[0], g1 = r[1];
      f2x F = g1.y;  // fc/2
      if (SAME) {
        float2 f = x_split(F);
        if (p == hole) { if (ow & 1) f.y = 0.0f; else f.x = 0.0f; }
        F = x_pack(f.x, f.y);
      }
      const f2x cs = x_fma(ux, g0.x, x_fma(uy, g0.y, x_mul(uz, g1.x)));
      const f2x hF = x_fma(cs, F, F);  // (1 + cos)/2 * fc_k
      const f2x tt = x_mul(hF, fj), ts = x_mul(hF, fs);
      f2x D = 0, B = 0;
#pragma unroll
      for (int c = 0; c < NCH; c++) {
        const ulonglong2 t = r[2 + c];
        const f2x be = beta[c];
        const float2 arg = x_split(x_mul(be, ts));
        const f2x E = x_pack(ex2_fast(arg.x), ex2_fast(arg.y));
        const f2x sum = x_fma(a1w[c], t.y, x_mul(a2w[c], t.x));             // w (S2 + S1)
        D = x_fma(x_mul(x_fma(be, tt, one2), E), sum, D);                   // w e^{bt} (1 + bt) (S1 + S2)
        B = x_fma(E, x_fma(b1w[c], t.y, x_mul(b2w[c], t.x)), B);            // w e^{bt} (a1 S2 + a2 S1)
      }
      // f_ij = cjk*u_k + (...)*u_j, the owner's factors applied at the end
      const f2x dk = x_mul(D, F);
      ax = x_fma(dk, g0.x, ax);
      ay = x_fma(dk, g0.y, ay);
      az = x_fma(dk, g1.x, az);
      ac = x_fma(cs, dk, ac);
      ah = x_fma(hF, x_fma(fj, B, D), ah);
    }
    const float2 vj = *reinterpret_cast<const float2*>(V + j);  // 1/r, dfc/dr
    const float cj = uj.w * vj.x;
    const float2 fx2 = x_split(ax), fy2 = x_split(ay), fz2 = x_split(az), c2 = x_split(ac), h2 = x_split(ah);
    const float asum = vj.y * (h2.x + h2.y) - cj * (c2.x + c2.y);
    float fx = cj * (fx2.x + fx2.y) + asum * uj.x, fy = cj * (fy2.x + fy2.y) + asum * uj.y,
          fz = cj * (fz2.x + fz2.y) + asum * uj.z;  // zero on lanes that are not active
    fix -= fx; fiy -= fy; fiz -= fz;
    if (NW == 1) {
      // the segments of an owner lie on consecutive lanes; its first lane of this round collects them.  (Shared float
      // atomics are compare-and-swap loops, S round trips each.)
      float gx = fx, gy = fy, gz = fz;
      for (int d = 1; d < S; d++) {
        const float tx = __shfl_down_sync(0xffffffffu, fx, d), ty = __shfl_down_sync(0xffffffffu, fy, d),
                    tz = __shfl_down_sync(0xffffffffu, fz, d);
        if (pos + d < S && lane + d < 32) { gx += tx; gy += ty; gz += tz; }
      }
      if (active && (pos == 0 || lane == 0)) {
        fo[j * 3] += gx; fo[j * 3 + 1] += gy; fo[j * 3 + 2] += gz;
      }
      __syncwarp();
    } else {
      flush_segments<float, NW>(oo, base, S, nseg, lane, fx, fy, fz, fo, part);
    }
  }
}

// Calls fn with the number of channels of this pass as a compile-time constant: every number in double precision,
// the next even one in fp32 (pairs of channels, the last one padded).
template <class T, class Fn>
__device__ __forceinline__ void by_channels(int nch, Fn&& fn) {
  if constexpr (sizeof(T) == 8) {
    switch (nch) {
      case 1: fn(std::integral_constant<int, 1>()); break;
      case 2: fn(std::integral_constant<int, 2>()); break;
      case 3: fn(std::integral_constant<int, 3>()); break;
      case 4: fn(std::integral_constant<int, 4>()); break;
      case 5: fn(std::integral_constant<int, 5>()); break;
      case 6: fn(std::integral_constant<int, 6>()); break;
      case 7: fn(std::integral_constant<int, 7>()); break;
      default: fn(std::integral_constant<int, 8>()); break;
    }
  } else {
    switch ((nch + 1) >> 1) {
      case 1: fn(std::integral_constant<int, 2>()); break;
      case 2: fn(std::integral_constant<int, 4>()); break;
      case 3: fn(std::integral_constant<int, 6>()); break;
      default: fn(std::integral_constant<int, 8>()); break;
    }
  }
}

// One block of NW warps per central atom.  VIR (force mode only) adds the virial; it is a template parameter so
// that the training step's force sweep does not carry its registers.  PACK: partner pairs (fp32 forces).
template <class T, int MODE, bool VIR, int NW, bool PACK>
__global__ void __launch_bounds__(32 * NW, (SweepMinBlocks<MODE, sizeof(T)>::value + NW - 1) / NW)
    k_sweep(ModelDev md, SweepArgs<T> a, SweepSmem L) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  typedef typename Vec4<T>::type T4;
  typedef typename Vec2<T>::type T2;
  constexpr bool IS_AF = (MODE == MODE_AF || MODE == MODE_AFV);
  constexpr int ES = (int)sizeof(T);
  constexpr int LANES = 32 * NW;
  const int lane = NW == 1 ? (int)threadIdx.x : (int)(threadIdx.x & 31), tid = threadIdx.x;
  int t, b, i;
  if (!locate_atom(md, a.nf, 1, 0, t, b, i)) return;
  const int N = md.N, nr = a.nr, nt = md.nt;
  const int Fr = md.Fr[t], Fa = md.Fa[t], Fmax = md.Fmax, Frmax = md.Frmax, Famax = md.Famax;
  const size_t gi = (size_t)b * N + i;
  const SparLayout& sl = a.sl;
  unsigned char* rowp = smem_raw + L.row;
  const T4* U = reinterpret_cast<const T4*>(rowp);
  const T4* V = reinterpret_cast<const T4*>(rowp + row_off_v(nr, ES));
  const int* ids = reinterpret_cast<const int*>(rowp + row_off_id(nr, ES));
  const int* hdr = reinterpret_cast<const int*>(rowp + row_off_hdr(nr, ES));
  unsigned char* spb = smem_raw + L.spar;
  const int* nact_s = reinterpret_cast<const int*>(spb);
  const int* nrad = nact_s + 8;
  const unsigned char* actc = spb + sl.actc;
  const T4* chq_all = reinterpret_cast<const T4*>(spb + sl.chq);
  const T2* chr_all = reinterpret_cast<const T2*>(spb + sl.chr);
  const T2* che_all = reinterpret_cast<const T2*>(spb + sl.che);
  const T4* rpar = reinterpret_cast<const T4*>(spb + sl.rpar);
  T4* tab4 = reinterpret_cast<T4*>(smem_raw + L.tab);
  T* xtra = reinterpret_cast<T*>(smem_raw + L.xtra);
  T* part = reinterpret_cast<T*>(smem_raw + L.part);
  T* acc = reinterpret_cast<T*>(smem_raw + L.acc);
  T* rsum = reinterpret_cast<T*>(smem_raw + L.rsum);
  T2* wch_all = reinterpret_cast<T2*>(smem_raw + L.wch);
  int* off = reinterpret_cast<int*>(smem_raw + L.red);  // [STAFB_MAX_TYPES + 1]
  T* et = reinterpret_cast<T*>(smem_raw + L.etab);
  const unsigned bar = smem_addr(smem_raw + L.mbar);
  // accumulator regions: the first nv entries are the d(AF)/d(alpha) row of the AFV mode
  const int ACC_A2 = 0;                      // [nt*Frmax]  alpha2b terms
  const int ACC_A3 = nt * Frmax;             // [C*3*Famax] alpha3b terms
  const int ACC_GN = ACC_A3 + md.C * 3 * Famax;  // [Famax]  fingerprints (AF, AFV) / gradnet (FGRAD)
  const int NACC = ACC_GN + Famax;

  // The neighbour record is at least two kernels old (it belongs to the neighbour kernel of this batch), and so is
  // the parameter block except in the fingerprint sweep, which directly follows k_prep.
  if (tid == 0) mbar_init(bar, 2);
  block_sync<NW>();
  if (tid == 0) {
    mbar_expect_tx(bar, (unsigned)a.row_stride);
    bulk_g2s(smem_addr(rowp), a.rows + gi * (size_t)a.row_stride, (unsigned)a.row_stride, bar);
    if (!IS_AF) {
      mbar_expect_tx(bar, (unsigned)sl.total);
      bulk_g2s(smem_addr(spb), a.spar + (size_t)t * a.spar_stride, (unsigned)sl.total, bar);
    }
  }
  if (MODE != MODE_FORCE)
    for (int q = tid; q < NACC; q += LANES) acc[q] = T(0);
  if (MODE != MODE_FORCE)
    for (int q = tid; q < nt * Frmax; q += LANES) rsum[q] = T(0);
  if (ES == 8 && tid < 16) et[tid] = (T)EXP16_TABLE[tid];
  chain_wait();
  if (IS_AF && tid == 0) {
    mbar_expect_tx(bar, (unsigned)sl.total);
    bulk_g2s(smem_addr(spb), a.spar + (size_t)t * a.spar_stride, (unsigned)sl.total, bar);
  }
  // what the preceding kernels produced for this atom, fetched while the copies are in flight
  const T* chrow = a.chan_in ? a.chan_in + gi * Fmax : nullptr;
  T fbx = T(0), fby = T(0), fbz = T(0);
  // dL/dF of one force component (the loss kernel's formula: Keras Huber(delta = 1) or squared error, mean)
  const T* fo_g = nullptr;
  const T* fl_g = nullptr;
  const T fscale = a.fscale;
  const bool hub = a.loss_kind == 0;
  auto fbar_of = [&](int q) -> T {
    const T e = fo_g[q] - fl_g[q];
    return fscale * (hub ? (e > T(1) ? T(1) : (e < T(-1) ? T(-1) : e)) : T(2) * e);
  };
  // dL/dW of this frame (virial loss of the energy + force + virial training, staf_model.py:313-384), kept behind
  // the group offsets
  T* wbs = reinterpret_cast<T*>(smem_raw + L.red) + 8;
  if (MODE == MODE_FGRAD) {
    fo_g = a.force + (size_t)b * a.nall * 3;
    fl_g = a.flab + (size_t)b * a.nall * 3;
    fbx = fbar_of(i * 3); fby = fbar_of(i * 3 + 1); fbz = fbar_of(i * 3 + 2);
    if (a.vacc) {
      // lane = slot: nine coalesced loads, nine warp sums
      double w = 0.0;
#pragma unroll
      for (int q = 0; q < 9; q++) {
        const double v = warp_sum(a.vacc[((size_t)b * 9 + q) * VIR_SLOTS + lane]);
        if (lane == q) w = v;
      }
      if (tid < 9) {
        const T e = (T)w - a.vlab[b * 9 + lane];
        wbs[lane] = a.vscale * (hub ? (e > T(1) ? T(1) : (e < T(-1) ? T(-1) : e)) : T(2) * e);
      }
    }
  }
  if (!mbar_wait(bar, 0)) {
    if (tid == 0) set_status(a.status, STAFB_ERR_STAGE_TIMEOUT);
    return;
  }
  int n = hdr[0];
  if (n > nr) n = nr;
  // first entry of every species' group (kept in shared memory like the counts, not in registers)
  if (tid == 0) {
    int o = 0;
    for (int q = 0; q < STAFB_MAX_TYPES; q++) {
      off[q] = o;
      o += (q < nt) ? hdr[2 + q] : 0;
    }
    off[STAFB_MAX_TYPES] = o;
  }
  block_sync<NW>();
  if (MODE == MODE_FGRAD) {
    // dF_k = Fbar_k - Fbar_i and its projection on the unit vector
    T4* dF = reinterpret_cast<T4*>(xtra);
    for (int k = tid; k < n; k += LANES) {
      const int id = ids[k];
      const T4 u = U[k];
      T4 d;
      d.x = fbar_of(id * 3) - fbx; d.y = fbar_of(id * 3 + 1) - fby; d.z = fbar_of(id * 3 + 2) - fbz;
      if (a.vacc) {
        // W_ab = -sum f_a r_b over the pairs: the virial's cotangent shifts the neighbour's force cotangent by
        // -(dL/dW) r with r = r_i - r_k (grad_force/rad/reforce.cu.cc:165-234, grad_force/ang/reforce.cu.cc:274-446)
        const T r = T(1) / V[k].x;
        const T rx = u.x * r, ry = u.y * r, rz = u.z * r;
        d.x -= wbs[0] * rx + wbs[1] * ry + wbs[2] * rz;
        d.y -= wbs[3] * rx + wbs[4] * ry + wbs[5] * rz;
        d.z -= wbs[6] * rx + wbs[7] * ry + wbs[8] * rz;
      }
      d.w = d.x * u.x + d.y * u.y + d.z * u.z;
      dF[k] = d;
    }
  }
  if (MODE == MODE_FORCE) {
    // channel weights 0.25 * e3 * netderiv of every (class, channel pair); the 0.5 of E = 0.5 sum e and the 0.5 of
    // the symmetrised pair sum
    for (int idx = tid; idx < md.ncls * sl.maxp; idx += LANES) {
      const int s = idx / sl.maxp, pr = idx - s * sl.maxp;
      T2 w = mk2(T(0), T(0));
      if (2 * pr < nact_s[s]) {
        const T2 ee = che_all[idx];
        w.x = T(0.25) * ee.x * chrow[Fr + actc[s * Famax + 2 * pr]];
        w.y = (2 * pr + 1 < nact_s[s]) ? T(0.25) * ee.y * chrow[Fr + actc[s * Famax + 2 * pr + 1]] : T(0);
      }
      wch_all[idx] = w;
    }
    // and 0.5 * e2 * netderiv of the radial ones
    for (int idx = tid; idx < nt * Frmax; idx += LANES) {
      const T4 rp = rpar[idx];
      rsum[idx] = rp.z != T(0) ? T(0.5) * rp.z * chrow[(int)rp.w] : T(0);
    }
  }
  block_sync<NW>();

  T fix = T(0), fiy = T(0), fiz = T(0);  // FORCE: force on the central atom
  // ------------------------------------------------------------------ radial part
  if (MODE == MODE_FORCE) {
    // g_k = 0.5 * sum_c netderiv_c e2 e^{alpha d}(1 + alpha d) * dd/dr * u_k  (force/rad/reforce.cu.cc:45-136)
    for (int k = tid; k < nr; k += LANES) {
      T gx = T(0), gy = T(0), gz = T(0);
      if (k < n) {
        int tk = 0;
#pragma unroll
        for (int q = 1; q < STAFB_MAX_TYPES; q++) tk += (q < nt && k >= off[q]) ? 1 : 0;
        const T4 u = U[k], v = V[k];
        const T dk = v.z;
        T w = T(0);
        const int c1 = (tk + 1) * Frmax;
        for (int c = tk * Frmax; c < c1; c++) {
          const T4 rp = rpar[c];
          if (rp.z == T(0)) break;  // compacted
          w += rsum[c] * (Ex<T>::f(rp.x * dk, et) * (T(1) + rp.y * dk));
        }
        const T g = w * v.w;
        gx = g * u.x; gy = g * u.y; gz = g * u.z;
        fix -= gx; fiy -= gy; fiz -= gz;
      }
      xtra[k * 3 + 0] = gx; xtra[k * 3 + 1] = gy; xtra[k * 3 + 2] = gz;
    }
  } else {
    // SEG lanes per active (neighbour species q, channel c) walk that species' neighbours, as many as there are lanes for
    // (several warps: each takes every NW-th neighbour), and add up by shuffles; the per-species sums of a channel are
    // combined through rsum[].  AF, AFV: fingerprints; FGRAD: gradnet; all but AF: alpha2b terms.
    // Inference and several warps per atom take one lane per row of rpar, active or not: their walks are short already and
    // the counting costs more than it saves (24,576-atom call 545 -> 549 us, 96-atom evaluation 56 -> 57.5 us with it).
    constexpr bool FLAT = MODE == MODE_AF || NW > 1;
    int items = nt * Frmax;
    if (!FLAT) {
      items = 0;
      for (int q = 0; q < nt; q++) items += nrad[q];
    }
    const int SEG = FLAT || items > 16 ? 1 : items > 10 ? 2 : items > 8 ? 3 : 4;
    for (int L0 = 0; L0 < items; L0 += 32) {
      const int it = L0 + (SEG == 1 ? lane : SEG == 2 ? lane >> 1 : SEG == 3 ? (lane * 21846) >> 16 : lane >> 2);
      const int sg = lane - (it - L0) * SEG;
      T gn = T(0), ga = T(0);
      int q = 0, c = 0;
      if (it < items) {
        c = it;
        if (FLAT) {
          q = it / Frmax;
          c = it - q * Frmax;
        } else {
          while (c >= nrad[q]) c -= nrad[q++];
        }
        const T4 rp = rpar[q * Frmax + c];
        c = (int)rp.w;
        const T als = rp.x, al = rp.y, alr = scale_rest(al, als);
        const int r0_ = off[q] + (NW == 1 ? sg : (tid >> 5) + NW * sg), r1_ = FLAT && rp.z == T(0) ? 0 : off[q + 1];
        const T4* dF = reinterpret_cast<const T4*>(xtra);
#pragma unroll 4
        for (int r = r0_; r < r1_; r += NW * SEG) {
          const T4 v = V[r];
          const T dk = v.z;
          const T ex = Ex<T>::f(sizeof(T) == 4 ? als * dk + alr * dk : als * dk, et);
          if (MODE == MODE_FGRAD) {
            const T qq = T(0.5) * v.w * dF[r].w;
            gn += qq * ex * (T(1) + al * dk);
            ga += qq * ex * dk * (T(2) + al * dk);
          } else {
            gn += dk * ex;
            ga += ex * dk * dk;
          }
        }
        gn *= rp.z;
        ga *= (MODE == MODE_FGRAD ? chrow[c] : T(1)) * rp.z;
      }
      T g1 = gn, a1 = ga;
      for (int d = 1; d < SEG; d++) {
        g1 += __shfl_down_sync(0xffffffffu, gn, d);
        if (MODE != MODE_AF) a1 += __shfl_down_sync(0xffffffffu, ga, d);
      }
      if (it < items && sg == 0 && (!FLAT || gn != T(0) || ga != T(0))) {
        if (NW == 1) {
          rsum[q * Frmax + c] = g1;
          if (MODE != MODE_AF) acc[ACC_A2 + q * Frmax + c] = a1;
        } else {
          atomicAdd(&rsum[q * Frmax + c], g1);
          if (MODE != MODE_AF) atomicAdd(&acc[ACC_A2 + q * Frmax + c], a1);
        }
      }
    }
    block_sync<NW>();
    if (MODE == MODE_FGRAD) {
      // the pair loops want W/4 and q/2 of every neighbour (pairs_unordered)
      T4* dF = reinterpret_cast<T4*>(xtra);
      for (int k = tid; k < n; k += LANES) {
        const T4 u = U[k];
        const T2 v = *reinterpret_cast<const T2*>(V + k);  // 1/r, dfc/dr
        const T4 d = dF[k];
        const T w = T(0.25) * u.w * v.x;
        T4 o;
        o.x = w * (d.x - d.w * u.x); o.y = w * (d.y - d.w * u.y); o.z = w * (d.z - d.w * u.z);
        o.w = T(0.5) * v.y * d.w;
        dF[k] = o;
      }
    }
    for (int c = tid; c < Fr; c += LANES) {
      T v = T(0);
      for (int q = 0; q < nt; q++) v += rsum[q * Frmax + c];
      a.out[gi * Fmax + c] = v;
    }
  }
  block_sync<NW>();

  // ------------------------------------------------------------------ angular part
  if constexpr (PACK) {
    float4* rec = reinterpret_cast<float4*>(smem_raw + L.tab);
    float4* cw = rec + FP_REC * fp_pairs(nr);  // the pass's channel weights and beta
    float2* beta = reinterpret_cast<float2*>(cw + FP_CH);
    // geometry of the angular neighbours in pairs
    for (int q = 0, p0 = 0; q < nt; q++) {
      const int n_ = hdr[6 + q], np_ = (n_ + 1) >> 1;
      for (int p = tid; p < np_; p += LANES) {
        const float4 u0 = U[off[q] + 2 * p];
        float4 u1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (2 * p + 1 < n_) u1 = U[off[q] + 2 * p + 1];
        rec[FP_REC * (p0 + p)] = make_float4(u0.x, u1.x, u0.y, u1.y);
        rec[FP_REC * (p0 + p) + 1] = make_float4(u0.z, u1.z, 0.5f * u0.w, 0.5f * u1.w);
      }
      p0 += np_;
    }
    block_sync<NW>();
    for (int ta = 0, pa = 0; ta < nt; ta++) {
      const int na_ = hdr[6 + ta], npa = (na_ + 1) >> 1;
      for (int tb = ta, pn = pa; tb < nt; tb++) {
        const int s = ta + tb, nb_ = hdr[6 + tb], npb = (nb_ + 1) >> 1, pb = pn;
        pn += npb;
        const bool same = (ta == tb);
        if ((same ? na_ < 2 : na_ * nb_ == 0) || s >= md.ncls) continue;
        const float* chq = reinterpret_cast<const float*>(chq_all + s * sl.maxp);
        const float* chr = reinterpret_cast<const float*>(chr_all + s * sl.maxp);
        const float* wch = reinterpret_cast<const float*>(wch_all + s * sl.maxp);
        const int nact = nact_s[s];
#pragma unroll 1
        for (int c0 = 0; c0 < nact; c0 += FP_CH) {
          const int nch = min(FP_CH, nact - c0);
          // tables of the pairs of the two species; x / nu by a reciprocal (exact: x < 2^10)
          const int nu = same ? npa : npa + npb, rcp = (int)__fdividef(1048576.0f, (float)nu) + 1;
          for (int x = tid; x < nu * nch; x += LANES) {
            const int c = (x * rcp) >> 20, r = x - c * nu, kp = r < npa ? pa + r : pb + (r - npa);
            const int ch = c0 + c, ci = (ch >> 1) * 4 + (ch & 1);
            const float4 g = rec[FP_REC * kp + 1];
            const float al1 = chq[ci] * (2.0f * Ex<float>::scale()), al2 = chq[ci + 2] * (2.0f * Ex<float>::scale());
            rec[FP_REC * kp + 2 + c] =
                make_float4(ex2_fast(al1 * g.z), ex2_fast(al1 * g.w), ex2_fast(al2 * g.z), ex2_fast(al2 * g.w));
          }
          if (tid < nch) {
            const int ch = c0 + tid, ci = (ch >> 1) * 4 + (ch & 1);
            const float w = wch[ch];
            cw[tid] = make_float4(w, chq[ci] * w, chq[ci + 2] * w, 0.0f);
            beta[tid] = mk2(chr[ch], chr[ch]);
          }
          block_sync<NW>();
          auto go = [&](auto tag) {
            constexpr int NCH = decltype(tag)::value;
            const f2x* be = reinterpret_cast<const f2x*>(beta);
            if (same) {
              pairs_force2<NCH, true, NW>(U, V, rec, be, cw, off[ta], pa, pa, na_, npa, tid, xtra, part, fix, fiy, fiz);
            } else {
#pragma unroll 1
              for (int pass = 0; pass < 2; pass++)
                pairs_force2<NCH, false, NW>(U, V, rec, be, cw, pass ? off[tb] : off[ta], pass ? pb : pa, pass ? pa : pb,
                                             pass ? nb_ : na_, pass ? npa : npb, tid, xtra, part, fix, fiy, fiz);
            }
          };
          switch (nch) {
            case 1: go(std::integral_constant<int, 1>()); break;
            case 2: go(std::integral_constant<int, 2>()); break;
            case 3: go(std::integral_constant<int, 3>()); break;
            case 4: go(std::integral_constant<int, 4>()); break;
            default: go(std::integral_constant<int, 5>()); break;
          }
          block_sync<NW>();  // the next pass rewrites the tables
        }
      }
      pa += npa;
    }
  }
  for (int ta = 0; ta < (PACK ? 0 : nt); ta++) {
    for (int tb = ta; tb < nt; tb++) {
      const int s = ta + tb;
      const int na_ = hdr[6 + ta], nb_ = hdr[6 + tb], oa = off[ta], ob = off[tb];
      const bool same = (ta == tb);
      const int np = same ? na_ * (na_ - 1) / 2 : na_ * nb_;
      if (np <= 0 || s >= md.ncls) continue;
      const int nact = nact_s[s];
      const int npair = (nact + 1) >> 1;
      for (int p0 = 0; p0 < npair; p0 += MAXP) {
        const int nchp = (npair - p0) < MAXP ? (npair - p0) : MAXP;
        const int nch = sizeof(T) == 4 ? 2 * nchp : ((nact - 2 * p0) < 2 * MAXP ? (nact - 2 * p0) : 2 * MAXP);
        const T4* chq = chq_all + s * sl.maxp + p0;
        const T2* chr = chr_all + s * sl.maxp + p0;
        // tables exp(a1*fc_k), exp(a2*fc_k) of the neighbours of the two species, all channel pairs of a
        // neighbour in flight together
        const int nu = same ? na_ : na_ + nb_;
        for (int r = tid; r < nu; r += LANES) {
          const int k = (r < na_) ? oa + r : ob + (r - na_);
          const T fck = U[k].w * Ex<T>::scale();
          const T2 f2 = mk2(fck, fck);
#pragma unroll
          for (int lp = 0; lp < MAXP; lp++) {
            if (lp < nchp) {
              const T4 q = chq[lp];
              const T2 e1 = p_ex(p_mul(mk2(q.x, q.y), f2), et), e2 = p_ex(p_mul(mk2(q.z, q.w), f2), et);
              T4 v;
              v.x = e1.x; v.y = e1.y; v.z = e2.x; v.w = e2.y;
              tab4[k * TSTR + lp] = v;
            }
          }
        }
        block_sync<NW>();
        if (MODE == MODE_FORCE) {
          const T2* wch = wch_all + s * sl.maxp + p0;
          const int npass = same ? 1 : 2;
          for (int pass = 0; pass < npass; pass++) {
            const int oo = pass == 0 ? oa : ob, op = pass == 0 ? ob : oa;
            const int no = pass == 0 ? na_ : nb_;
            const int npt = same ? na_ - 1 : (pass == 0 ? nb_ : na_);
            auto go = [&](auto tag) {
              constexpr int NCH = decltype(tag)::value;
              if (same)
                pairs_force<T, NCH, true, NW>(U, V, tab4, chq, chr, wch, et, oo, op, no, npt, tid, xtra, part, fix, fiy, fiz);
              else
                pairs_force<T, NCH, false, NW>(U, V, tab4, chq, chr, wch, et, oo, op, no, npt, tid, xtra, part, fix, fiy, fiz);
            };
            by_channels<T>(nch, go);
          }
        } else {
          // per-lane sums, then the transposing butterfly: lane L ends up with the total of value index L (or
          // L >> 1, L >> 2 when fewer values are carried).  Value index = 8*lp + 4*h + v for channel 2*lp + h of
          // the chunk and term v (0 fingerprint / gradnet, 1..3 alpha1, alpha2, beta); AF carries v = 0 only,
          // index 2*lp + h.
          const T4* dF = reinterpret_cast<const T4*>(xtra);
          T tot = T(0);
          int vidx = -1;  // value index this lane holds after the reduction (-1: none)
          auto run = [&](auto nch_tag) {
            constexpr int NCH = decltype(nch_tag)::value, NCHP = (NCH + 1) / 2;
            T2 r0[NCHP], r1[NCHP], r2[NCHP], r3[NCHP];
            if (same)
              pairs_unordered<T, MODE, NCH, true, NW>(U, V, dF, tab4, nr, chq, chr, et, oa, ob, na_, nb_, tid, r0, r1, r2,
                                                      r3);
            else
              pairs_unordered<T, MODE, NCH, false, NW>(U, V, dF, tab4, nr, chq, chr, et, oa, ob, na_, nb_, tid, r0, r1, r2,
                                                       r3);
            if (MODE == MODE_AF) {
              constexpr int NV = NCHP == 1 ? 2 : (NCHP == 2 ? 4 : 8);
              T v[NV];
#pragma unroll
              for (int q = 0; q < NV; q++) v[q] = T(0);
#pragma unroll
              for (int lp = 0; lp < NCHP; lp++) { v[2 * lp] = r0[lp].x; v[2 * lp + 1] = r0[lp].y; }
              tot = multi_reduce<T, NV>(v, lane);
              constexpr int SH = NV == 2 ? 4 : (NV == 4 ? 3 : 2);  // log2(32 / NV)
              vidx = ((lane & ((1 << SH) - 1)) == 0) ? (lane >> SH) : -1;
              if (vidx >= 0) vidx = 8 * (vidx >> 1) + 4 * (vidx & 1);  // as (lp, h, v = 0)
            } else {
              constexpr int NV = NCHP == 1 ? 8 : (NCHP == 2 ? 16 : 32);
              T v[NV];
#pragma unroll
              for (int q = 0; q < NV; q++) v[q] = T(0);
#pragma unroll
              for (int lp = 0; lp < NCHP; lp++) {
                v[8 * lp] = r0[lp].x; v[8 * lp + 1] = r1[lp].x; v[8 * lp + 2] = r2[lp].x; v[8 * lp + 3] = r3[lp].x;
                v[8 * lp + 4] = r0[lp].y; v[8 * lp + 5] = r1[lp].y; v[8 * lp + 6] = r2[lp].y; v[8 * lp + 7] = r3[lp].y;
              }
              tot = multi_reduce<T, NV>(v, lane);
              constexpr int SH = NV == 8 ? 2 : (NV == 16 ? 1 : 0);
              vidx = ((lane & ((1 << SH) - 1)) == 0) ? (lane >> SH) : -1;
            }
          };
          by_channels<T>(nch, run);
          if (vidx >= 0) {
            const int lp = vidx >> 3, h = (vidx >> 2) & 1, v = vidx & 3;
            const int slot = 2 * (p0 + lp) + h;
            if (lp < nchp && slot < nact) {
              const int c = actc[s * Famax + slot];
              const T2 ee = che_all[s * sl.maxp + p0 + lp];
              const T cf = T(0.5) * (h ? ee.y : ee.x);
              if (v == 0) acc_add<NW>(&acc[ACC_GN + c], cf * tot);
              else if (MODE != MODE_AF) {
                const T hn = MODE == MODE_FGRAD ? cf * chrow[Fr + c] : cf;
                acc_add<NW>(&acc[ACC_A3 + (s * Famax + c) * 3 + (v - 1)], hn * tot);
              }
            }
          }
        }
        block_sync<NW>();  // the next chunk rewrites the tables
      }
    }
  }
  block_sync<NW>();

  // ------------------------------------------------------------------ write-back
  if (IS_AF) {
    for (int c = tid; c < Fa; c += LANES) a.out[gi * Fmax + Fr + c] = acc[ACC_GN + c];
    for (int c = Fr + Fa + tid; c < Fmax; c += LANES) a.out[gi * Fmax + c] = T(0);
    if (MODE == MODE_AFV) {
      T* vr = a.vout + gi * a.nv;
      for (int q = tid; q < a.nv; q += LANES) vr[q] = acc[q];
    }
  } else if (MODE == MODE_FORCE) {
    T* fbo = a.out + (size_t)b * a.nall * 3;
    for (int q = tid; q < 3 * n; q += LANES) atomicAdd(fbo + (size_t)ids[q / 3] * 3 + (q % 3), xtra[q]);
    fix = warp_sum(fix); fiy = warp_sum(fiy); fiz = warp_sum(fiz);
    if (lane == 0) {
      atomicAdd(fbo + (size_t)i * 3 + 0, fix);
      atomicAdd(fbo + (size_t)i * 3 + 1, fiy);
      atomicAdd(fbo + (size_t)i * 3 + 2, fiz);
    }
    if (VIR) {
      // W_ab -= g_a * r_b with g the force this centre puts on neighbour k and r = r_i - r_k
      // (force/rad/reforce.cu.cc:174-287, force/ang/reforce.cu.cc:269-457 of the reference)
      // one row of W at a time keeps the epilogue's register footprint below the main loop's
#pragma unroll 1
      for (int c = 0; c < 3; c++) {
        T w0 = T(0), w1 = T(0), w2 = T(0);
        for (int k = tid; k < n; k += LANES) {
          const T4 u = U[k];
          const T g = xtra[k * 3 + c] / V[k].x;  // g_a * |r|
          w0 -= g * u.x; w1 -= g * u.y; w2 -= g * u.z;
        }
        w0 = warp_sum(w0); w1 = warp_sum(w1); w2 = warp_sum(w2);
        if (lane == 0) {
          double* vs = a.vir + ((size_t)b * 9 + c * 3) * VIR_SLOTS + (i & (VIR_SLOTS - 1));
          atomicAdd(vs, (double)w0);
          atomicAdd(vs + VIR_SLOTS, (double)w1);
          atomicAdd(vs + 2 * VIR_SLOTS, (double)w2);
        }
      }
    }
  } else {  // FGRAD
    for (int c = tid; c < Fa; c += LANES) a.out[gi * Fmax + Fr + c] = acc[ACC_GN + c];
    for (int c = Fr + Fa + tid; c < Fmax; c += LANES) a.out[gi * Fmax + c] = T(0);
    if (a.grad) {
      T* g2 = a.grad + md.off_a2[t];
      for (int q = 0; q < nt; q++)
        for (int x = tid; x < nrad[q]; x += LANES) {
          const int c = (int)rpar[q * Frmax + x].w;
          atomicAdd(g2 + q * Fr + c, acc[ACC_A2 + q * Frmax + c]);
        }
      T* g3 = a.grad + md.off_a3[t];
      for (int s = 0; s < md.ncls; s++)
        for (int x = tid; x < 3 * nact_s[s]; x += LANES) {
          const int slot = x / 3, comp = x - 3 * slot, c = actc[s * Famax + slot];
          const T v = acc[ACC_A3 + (s * Famax + c) * 3 + comp];
          if (v != T(0)) atomicAdd(g3 + (s * Fa + c) * 3 + comp, v);
        }
    }
  }
}
