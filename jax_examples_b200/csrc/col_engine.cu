// Column engine for the high angular-momentum J/K classes (L >= 5).
//
// One warp evaluates one contracted shell quartet (ab|cd) of a class fixed at
// compile time.  Per primitive quartet:
//   * lanes 0..2 build the bra E coefficients of one axis each (once per bra
//     primitive pair), lanes 3..5 the ket E (with (-1)^t), lanes 0..L the
//     Boys values F_m(T) times the prefactor, all into the warp's slice of
//     shared memory; the R_tuv recursion then runs in shared memory, lanes
//     parallel over the entries of one total order;
//   * lane h (and h + 32) owns a bra Hermite index: it reads R_{h+k} for every
//     ket Hermite index k and turns the ket side Cartesian, X[cd][h], one axis
//     at a time (hermite_to_cart), summed over the ket primitives.
// Per bra primitive, lane cd reads its row X[cd][.] and turns the bra side
// Cartesian into block[ab][cd].  The earlier form had lane = cd throughout and
// summed over all Hermite pairs with one shared-memory read per multiply-add.
// Digestion into J/K is the warp engine's (warp_digest_jk).
#include "axis_transform.cuh"

namespace jqc {

template <typename T, int LA, int LB, int LC, int LD>
struct ColSmem {
  static constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
  static constexpr int NAB = ncart(LA) * ncart(LB), NCD = ncart(LC) * ncart(LD);
  static constexpr int kRow = nherm(LAB) | 1;  // odd: the rows of X on different banks
  T Eb[3][LA + 1][LB + 1][LAB + 1];
  T Fk[3][LC + 1][LD + 1][LCD + 1];
  T R[nherm(L)];
  T Rn[L + 1];
  T X[NCD * kRow];
  T blk[NAB * NCD];
};

constexpr int kColWarps = 4;
constexpr int kColSumWords = (HermSumTable::N * HermSumTable::N + 3) / 4;

// Bra E coefficients of one bra primitive pair (lanes 0..2, one axis each).
// The caller synchronises the warp before (earlier readers) and after.
template <typename T, int LA, int LB, int LC, int LD>
__device__ __forceinline__ void col_set_bra(ColSmem<T, LA, LB, LC, LD>* sm, const typename PPType<T>::type& bp,
                                            Vec3<T> A, Vec3<T> B, int lane) {
  if (lane == 0) ecoef_compute<T, LA, LB, false>(sm->Eb[0], bp.Px - A.x, bp.Px - B.x, bp.h);
  if (lane == 1) ecoef_compute<T, LA, LB, false>(sm->Eb[1], bp.Py - A.y, bp.Py - B.y, bp.h);
  if (lane == 2) ecoef_compute<T, LA, LB, false>(sm->Eb[2], bp.Pz - A.z, bp.Pz - B.z, bp.h);
}

// One primitive quartet's X[cd][h] into sm->X (added to it unless `first`); all
// lanes call with the same arguments and leave the warp synchronised.  `sum`:
// kHermSum in shared memory.
template <typename T, int LA, int LB, int LC, int LD>
__device__ __forceinline__ void col_add_prim(ColSmem<T, LA, LB, LC, LD>* sm, const typename PPType<T>::type& bp,
                                             const typename PPType<T>::type& kp, Vec3<T> C, Vec3<T> D,
                                             const T* __restrict__ tab, const unsigned char* sum, bool first,
                                             int lane) {
  using S = ColSmem<T, LA, LB, LC, LD>;
  constexpr int L = S::L, NH = nherm(S::LAB), NK = nherm(S::LCD);
  if (lane == 3) ecoef_compute<T, LC, LD, true>(sm->Fk[0], kp.Px - C.x, kp.Px - D.x, kp.h);
  if (lane == 4) ecoef_compute<T, LC, LD, true>(sm->Fk[1], kp.Py - C.y, kp.Py - D.y, kp.h);
  if (lane == 5) ecoef_compute<T, LC, LD, true>(sm->Fk[2], kp.Pz - C.z, kp.Pz - D.z, kp.h);
  const T r = fast_rsqrt(bp.p + kp.p);
  const T rho = bp.p * kp.p * (r * r);
  const T X = bp.Px - kp.Px, Y = bp.Py - kp.Py, Z = bp.Pz - kp.Pz;
  const T tb = rho * (X * X + Y * Y + Z * Z);
  if (lane <= L) {
    T pref = T(4.0 * kTwoPi25) * bp.K * kp.K * (bp.h * kp.h) * r;
    const T m2rho = T(-2) * rho;
    for (int k = 0; k < lane; ++k) pref *= m2rho;
    sm->Rn[lane] = pref * boys_single<T>(tb, lane, tab);
  }
  __syncwarp();
  warp_hermite_R<T, L>(sm->R, sm->Rn, X, Y, Z, lane);
  for (int h = lane; h < NH; h += 32) {
    T rk[NK];
    static_for<NK>([&](auto k_) {
      constexpr int k = decltype(k_)::value;
      rk[k] = sm->R[sum[k * HermSumTable::N + h]];
    });
    hermite_to_cart<LC, LD, 0, LC + 1>(rk, sm->Fk, [&](auto cd_, T v) {
      T* x = sm->X + decltype(cd_)::value * S::kRow + h;
      *x = first ? v : *x + v;
    });
  }
  __syncwarp();
}

// Accumulates block[ab][cd] of one shell quartet over bra primitive pairs
// [0, nbra) and ket primitive pairs [0, nket) into sm->blk (zeroed here).
template <typename T, int LA, int LB, int LC, int LD>
__device__ __forceinline__ void col_quartet(ColSmem<T, LA, LB, LC, LD>* sm, const typename PPType<T>::type* bra,
                                            int nbra, Vec3<T> A, Vec3<T> B, const typename PPType<T>::type* ket,
                                            int nket, Vec3<T> C, Vec3<T> D, const T* __restrict__ tab,
                                            const unsigned char* sum, int lane) {
  using S = ColSmem<T, LA, LB, LC, LD>;
  using PPT = typename PPType<T>::type;
  constexpr int NH = nherm(S::LAB), NCD = S::NCD;
  for (int i = lane; i < S::NAB * S::NCD; i += 32) sm->blk[i] = T(0);
  for (int ip = 0; ip < nbra; ++ip) {
    const PPT bp = ld_pp(bra + ip);
    __syncwarp();
    col_set_bra<T, LA, LB, LC, LD>(sm, bp, A, B, lane);
    for (int iq = 0; iq < nket; ++iq) {
      const PPT kp = ld_pp(ket + iq);
      col_add_prim<T, LA, LB, LC, LD>(sm, bp, kp, C, D, tab, sum, iq == 0, lane);
    }
    if (nket == 0) continue;
    for (int c = lane; c < NCD; c += 32) {
      T x[NH];
      static_for<NH>([&](auto h_) { x[decltype(h_)::value] = sm->X[c * S::kRow + decltype(h_)::value]; });
      hermite_to_cart<LA, LB, 0, LA + 1>(x, sm->Eb,
                                         [&](auto ab_, T v) { sm->blk[decltype(ab_)::value * NCD + c] += v; });
    }
  }
  __syncwarp();
}

// Resident blocks a multiprocessor the register allocation aims at: three (168
// registers, 12 warps) for the FP64 (dd|dp), 270 -> 223 us in a full (H2O)16
// build (four: 218, but 416 bytes spilled and the whole build slower); (dd|dd)
// loses to its spills (74 -> 91 us).  Against the form with lane = cd throughout
// and dense sums: (dd|dp) 301 -> 223 us, (dd|dd) 83 -> 74.  About 5500 warp
// instructions a quartet, a quarter of them the digestion, at 0.3 an issue
// slot: bound by latency and by the second lane pass for 35 Hermite functions.
template <typename T>
__host__ __device__ constexpr int col_min_blocks(int lc, int ld) {
  return sizeof(T) == 8 && lc == 2 && ld == 1 ? 3 : 1;
}

template <typename T, int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(32 * kColWarps, col_min_blocks<T>(LC, LD)) col_jk_kernel(const JKParams prm) {
  using S = ColSmem<T, LA, LB, LC, LD>;
  using PPT = typename PPType<T>::type;
  extern __shared__ __align__(16) unsigned char col_smraw[];
  S* sm = reinterpret_cast<S*>(col_smraw) + (threadIdx.x >> 5);
  unsigned char* sum = col_smraw + kColWarps * sizeof(S);
  for (int i = int(threadIdx.x); i < kColSumWords; i += int(blockDim.x))
    reinterpret_cast<unsigned*>(sum)[i] = __ldg(reinterpret_cast<const unsigned*>(kHermSum.v) + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= prm.n_tasks) return;
  if (prm.items != nullptr) {  // compacted work: the grid covers the whole list
    if (warp >= *prm.n_items) return;
    warp = prm.items[warp];
  }
  const Task task = prm.tasks[warp];
  const ShellPair bp = prm.pairs[task.bra];
  const PPT* pp = static_cast<const PPT*>(prm.pp);
  const T* tab = static_cast<const T*>(prm.boys);
  const double* ctr = prm.centres;
  const Vec3<T> A{T(ctr[3 * bp.a]), T(ctr[3 * bp.a + 1]), T(ctr[3 * bp.a + 2])};
  const Vec3<T> B{T(ctr[3 * bp.b]), T(ctr[3 * bp.b + 1]), T(ctr[3 * bp.b + 2])};
  for (int kk = 0; kk < int(task.nket); ++kk) {
    const int kidx = task.ket0 + kk;
    const ShellPair kp = prm.pairs[kidx];
    if (prm.dmax_top != nullptr && float(bp.Q) * float(kp.Q) * (2.f * *prm.dmax_top) < prm.dens_tau)
      continue;  // below the bound for any density block
    if (prm.dmax != nullptr) {
      const float* dm = prm.dmax;
      const int ns = prm.n_shell;
      float m = fmaxf(2.f * dm[bp.a * ns + bp.b], 2.f * dm[kp.a * ns + kp.b]);
      m = fmaxf(m, fmaxf(dm[bp.a * ns + kp.a], dm[bp.a * ns + kp.b]));
      m = fmaxf(m, fmaxf(dm[bp.b * ns + kp.a], dm[bp.b * ns + kp.b]));
      if (float(bp.Q) * float(kp.Q) * m < prm.dens_tau) continue;  // uniform over the warp
    }
    const Vec3<T> C{T(ctr[3 * kp.a]), T(ctr[3 * kp.a + 1]), T(ctr[3 * kp.a + 2])};
    const Vec3<T> Dv{T(ctr[3 * kp.b]), T(ctr[3 * kp.b + 1]), T(ctr[3 * kp.b + 2])};
    const int p0 = task.flags & 0xffff, p1 = task.flags >> 16;
    col_quartet<T, LA, LB, LC, LD>(sm, pp + bp.pp + p0, p1 - p0, A, B, pp + kp.pp, kp.npp, C, Dv, tab, sum, lane);
    double s = 1.0;
    if (bp.diag()) s *= 0.5;
    if (kp.diag()) s *= 0.5;
    if (task.bra == kidx) s *= 0.5;
    warp_digest_jk<T>(prm, sm->blk, ncart(LA), ncart(LB), ncart(LC), ncart(LD), prm.ao[bp.a], prm.ao[bp.b],
                      prm.ao[kp.a], prm.ao[kp.b], s, lane);
    __syncwarp();
  }
}

template <typename T, int LA, int LB, int LC, int LD>
static cudaError_t launch_col_jk_class(const JKParams& p, cudaStream_t s) {
  if (p.n_tasks == 0) return cudaSuccess;
  const size_t sm = kColWarps * sizeof(ColSmem<T, LA, LB, LC, LD>) + 4 * kColSumWords;
  // on every launch: the limit is the current device's, and contexts of several
  // devices and threads come here
  cudaError_t e = cudaFuncSetAttribute(col_jk_kernel<T, LA, LB, LC, LD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sm);
  if (e != cudaSuccess) return e;
  const unsigned grid = (unsigned)((p.n_tasks + kColWarps - 1) / kColWarps);
  col_jk_kernel<T, LA, LB, LC, LD><<<grid, 32 * kColWarps, sm, s>>>(p);
  return cudaGetLastError();
}

// Classes with a column-engine kernel.
#define JQC_FOR_COL_CLASSES(X) \
  X(12, 2, 1, 1, 1)            \
  X(13, 2, 1, 2, 0)            \
  X(14, 2, 1, 2, 1)            \
  X(16, 2, 2, 1, 0)            \
  X(17, 2, 2, 1, 1)            \
  X(18, 2, 2, 2, 0)            \
  X(19, 2, 2, 2, 1)            \
  X(20, 2, 2, 2, 2)

bool has_col_class(int qc) {
  switch (qc) {
#define X(Q, A, B, C, D) case Q:
    JQC_FOR_COL_CLASSES(X)
#undef X
    return true;
    default:
      return false;
  }
}

cudaError_t launch_col_jk(int qc, bool fp32, const JKParams& p, cudaStream_t s) {
  switch (qc) {
#define X(Q, A, B, C, D) \
  case Q:                \
    return fp32 ? launch_col_jk_class<float, A, B, C, D>(p, s) : launch_col_jk_class<double, A, B, C, D>(p, s);
    JQC_FOR_COL_CLASSES(X)
#undef X
    default:
      return cudaErrorNotSupported;
  }
}

}  // namespace jqc
