// McMurchie-Davidson machinery for contracted shell quartets on the device.
//
// The algorithm is the reference's (jax_qc/integrals/obara_saika.py:227-332,
// mcmurchie_davidson.py:60-172):
//   (ab|cd) = 2 pi^{5/2} / (p q sqrt(p+q)) K_AB K_CD
//             sum_{tuv} E^{ab}_{tuv} sum_{t'u'v'} (-1)^{t'+u'+v'} E^{cd}_{t'u'v'}
//             R_{t+t', u+u', v+v'}(rho, P-Q)
// restructured for registers: everything is unrolled at compile time for one
// angular class (LA LB | LC LD); the R_tuv^n recursion runs in place over n
// (one array of C(L+3,3) values); the Hermite contraction is done in two
// stages, first over the ket Hermite index into X_tuv for one ket Cartesian
// pair, then over the bra Hermite index into the output block.
#pragma once

#include "boys.cuh"
#include "common.cuh"

namespace jqc {

// One primitive pair of a shell pair (a, b): p = alpha + beta,
// P = (alpha A + beta B) / p, K = exp(-alpha beta |AB|^2 / p) c_a c_b,
// h = 1/(2p) (kept so no kernel divides by p).  32-byte aligned: the records
// live in cudaMalloc'd arrays and are read with 32-byte vector loads.
struct __align__(32) PrimPair {
  double p, h, Px, Py, Pz, K, alpha, beta;
};
struct __align__(32) PrimPairF {
  float p, h, Px, Py, Pz, K, alpha, beta;
};
static_assert(sizeof(PrimPair) == 64 && sizeof(PrimPairF) == 32, "primitive-pair records");

// 32-byte vector loads of a primitive-pair record through the read-only path
// (global memory only; records built in registers/local memory are read
// with plain loads, see quartet_accumulate's GLOBAL_PP).
__device__ __forceinline__ PrimPair ld_pp(const PrimPair* q) {
  const double* v = reinterpret_cast<const double*>(q);
  PrimPair r;
  ldg32B(v, r.p, r.h, r.Px, r.Py);
  ldg32B(v + 4, r.Pz, r.K, r.alpha, r.beta);
  return r;
}
__device__ __forceinline__ PrimPairF ld_pp(const PrimPairF* q) {
  float v[8];
  ldg32B(reinterpret_cast<const float*>(q), v);
  return PrimPairF{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]};
}
template <typename T>
struct PPType;
template <>
struct PPType<double> {
  using type = PrimPair;
};
template <>
struct PPType<float> {
  using type = PrimPairF;
};

// The same primitive pair as the register kernels read it: everything relative
// to the shell pair's own centres.  t = beta / p, so P - A = t (B - A) and
// P - B = (P - A) - (B - A); W = K h sqrt(8 pi^{5/2}), so the prefactor of a
// primitive quartet is W_ab W_cd / sqrt(p + q).  A lane's load writes its full
// width back to the registers whether or not the address is shared (128 bytes
// a cycle and SM), and that data path, 80% busy, bound the low-L kernels: 32
// bytes a primitive pair instead of 64 is what this record is for ((H2O)16 full
// build: (ss|ss) 595 -> 550 us, (ds|ss) 522 -> 494, (ps|ps) 449 -> 430; the
// closed-form tail of boys_hermite took them to 522, 474, 421).  Distances
// formed from differences of centres are also no less accurate than those of
// absolute positions (in FP32 markedly more).
struct __align__(32) PrimRec {
  double p, t, W, h;
};
struct __align__(16) PrimRecF {
  float p, t, W, h;
};
static_assert(sizeof(PrimRec) == 32 && sizeof(PrimRecF) == 16, "primitive-pair records");

__device__ __forceinline__ PrimRec ld_rec(const PrimRec* q) {
  PrimRec r;
  ldg32B(reinterpret_cast<const double*>(q), r.p, r.t, r.W, r.h);
  return r;
}
__device__ __forceinline__ PrimRecF ld_rec(const PrimRecF* q) {
  const float4 v = __ldg(reinterpret_cast<const float4*>(q));
  return PrimRecF{v.x, v.y, v.z, v.w};
}
template <typename T>
struct RecType;
template <>
struct RecType<double> {
  using type = PrimRec;
};
template <>
struct RecType<float> {
  using type = PrimRecF;
};

// Shell pair (a, b) with la >= lb.  pp/npp index its primitive pairs
// (contiguous); record i of the pair is at rec + i * stride().  Inside a block
// of pairs (same class and npp) the records are primitive-major, so the lanes
// of a warp, consecutive ket pairs, read consecutive records.
struct __align__(16) ShellPair {
  int a, b, pp, npp;
  double Q;    // Schwarz bound sqrt(max (ab|ab))
  int rec;
  unsigned stride_diag;
  __host__ __device__ int stride() const { return int(stride_diag >> 1); }
  __host__ __device__ bool diag() const { return (stride_diag & 1u) != 0u; }  // a == b
};

// Work item: one bra pair against a run of at most 32 consecutive ket pairs.
// flags: the bra's primitive pairs [flags & 0xffff, flags >> 16); q0, q1: the
// kets' primitive pairs (register kernels only; the other engines' tasks have
// them all).
struct __align__(16) Task {
  static constexpr unsigned kAllPrims = 4095;
  int bra, ket0;
  unsigned nket : 8, q0 : 12, q1 : 12;
  int flags;
  __host__ __device__ int ket_begin() const { return int(q0); }
  __host__ __device__ int ket_end(int npp) const { return q1 == kAllPrims ? npp : int(q1); }
};
static_assert(sizeof(Task) == 16, "tasks are read as one vector");

constexpr double kTwoPi25 = 34.986836655249725693;  // 2 pi^{5/2}
// sqrt(8 pi^{5/2}) in two parts: the first alone is 6.1e-17 off, which both
// sides of a quartet share (1.2e-16 in every integral, always the same way).
constexpr double kSqrt8Pi25 = 11.8299343455912257556, kSqrt8Pi25Lo = -7.1877868215575968e-16;

// ---------------------------------------------------------------- E coeffs

// E^{ij}_t along one axis for i <= LA, j <= LB (E^{00}_0 = 1), by
//   E^{i+1,j}_t = E^{ij}_{t-1}/(2p) + X_PA E^{ij}_t + (t+1) E^{ij}_{t+1}
//   E^{i,j+1}_t = E^{ij}_{t-1}/(2p) + X_PB E^{ij}_t + (t+1) E^{ij}_{t+1}
// (mcmurchie_davidson.py:60-108).  With SIGN the coefficients carry
// (-1)^t (the ket side of the contraction).
template <typename T, int LA, int LB>
using EArr = T (*)[LB + 1][LA + LB + 1];

template <typename T, int LA, int LB, bool SIGN>
__device__ __forceinline__ void ecoef_compute(EArr<T, LA, LB> e, T pa, T pb, T inv2p) {
  e[0][0][0] = T(1);
  static_for<LA>([&](auto ii) {
    constexpr int i = decltype(ii)::value;
    static_for<i + 2>([&](auto tt) {
      constexpr int t = decltype(tt)::value;
      T v = T(0);
      if constexpr (t <= i) v = pa * e[i][0][t];
      if constexpr (t >= 1) v += inv2p * e[i][0][t - 1];
      if constexpr (t + 1 <= i) v += T(t + 1) * e[i][0][t + 1];
      e[i + 1][0][t] = v;
    });
  });
  static_for<LB>([&](auto jj) {
    constexpr int j = decltype(jj)::value;
    static_for<LA + 1>([&](auto ii) {
      constexpr int i = decltype(ii)::value;
      static_for<i + j + 2>([&](auto tt) {
        constexpr int t = decltype(tt)::value;
        T v = T(0);
        if constexpr (t <= i + j) v = pb * e[i][j][t];
        if constexpr (t >= 1) v += inv2p * e[i][j][t - 1];
        if constexpr (t + 1 <= i + j) v += T(t + 1) * e[i][j][t + 1];
        e[i][j + 1][t] = v;
      });
    });
  });
  if constexpr (SIGN) {
    static_for<LA + 1>([&](auto ii) {
      static_for<LB + 1>([&](auto jj) {
        constexpr int i = decltype(ii)::value, j = decltype(jj)::value;
        static_for<(i + j + 1) / 2>([&](auto kk) {
          constexpr int t = 2 * decltype(kk)::value + 1;
          e[i][j][t] = -e[i][j][t];
        });
      });
    });
  }
}

// ---------------------------------------------------------------- R_tuv

// In-place R recursion.  On entry Rn[n] = pref * (-2 rho)^n F_n(T), n <= L.
// On exit R[herm_index(t,u,v)] = pref * R^0_{tuv} for t+u+v <= L.
// Level n is built from level n+1 by t/u/v raising (Helgaker 9.9.18-20);
// within a level, higher total orders are written first so every read sees
// level n+1 values.
template <typename T, int L>
__device__ __forceinline__ void hermite_R(T (&R)[nherm(L)], const T (&Rn)[L + 1], T X, T Y, T Z) {
  R[0] = Rn[L];
  static_for<L>([&](auto nn) {
    constexpr int n = L - 1 - decltype(nn)::value;
    static_for<L - n>([&](auto ss) {
      constexpr int s = L - n - decltype(ss)::value;
      static_for<ncart(s)>([&](auto kk) {
        constexpr int k = decltype(kk)::value;
        constexpr int t = cart_lx(s, k), u = cart_ly(s, k), v = s - t - u;
        T val;
        if constexpr (t > 0) {
          val = X * R[herm_index(t - 1, u, v)];
          if constexpr (t > 1) val += T(t - 1) * R[herm_index(t - 2, u, v)];
        } else if constexpr (u > 0) {
          val = Y * R[herm_index(t, u - 1, v)];
          if constexpr (u > 1) val += T(u - 1) * R[herm_index(t, u - 2, v)];
        } else {
          val = Z * R[herm_index(t, u, v - 1)];
          if constexpr (v > 1) val += T(v - 1) * R[herm_index(t, u, v - 2)];
        }
        R[herm_index(t, u, v)] = val;
      });
    });
    R[0] = Rn[n];
  });
}

// ------------------------------------------------------------ quartet core

template <int LA, int LB, int LC, int LD, int NS, int PART>
struct QCfg {
  static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  static constexpr int NAB = NA * NB, NCD = NC * ND;
  static constexpr int CDP = (NCD + NS - 1) / NS;  // ket Cartesian pairs per part
  static constexpr int CD0 = PART * CDP;
  static constexpr int NCDP = (CD0 >= NCD) ? 0 : ((CD0 + CDP <= NCD) ? CDP : NCD - CD0);
  static constexpr int L = LA + LB + LC + LD;
  static constexpr int LAB = LA + LB;
};

template <typename T>
struct Vec3 {
  T x, y, z;
};

__device__ __forceinline__ double fast_rsqrt(double x) { return rsqrt(x); }
__device__ __forceinline__ float fast_rsqrt(float x) { return rsqrtf(x); }

// R of one primitive quartet from the exponents, W = W_ab W_cd and P - Q.
template <typename T, int L>
__device__ __forceinline__ void prim_quartet_R(T p, T q, T W, T PQx, T PQy, T PQz, const T* __restrict__ boys_tab,
                                               T (&R)[nherm(L)]) {
  T Rn[L + 1];
  boys_hermite<T, L>(p * q, p + q, PQx * PQx + PQy * PQy + PQz * PQz, W, boys_tab, Rn);
  hermite_R<T, L>(R, Rn, PQx, PQy, PQz);
}
// The same from two full primitive-pair records (1/(pq) = 4 h_p h_q).
template <typename T, int L, typename PPT>
__device__ __forceinline__ void prim_quartet_R(const PPT& bp, const PPT& kp, const T* __restrict__ boys_tab,
                                               T (&R)[nherm(L)]) {
  prim_quartet_R<T, L>(bp.p, kp.p, T(4.0 * kTwoPi25) * T(bp.K) * T(kp.K) * (T(bp.h) * T(kp.h)), bp.Px - kp.Px,
                       bp.Py - kp.Py, bp.Pz - kp.Pz, boys_tab, R);
}

// Classes whose bra angular sum is at most this loop over ket primitives
// outermost (see quartet_accumulate) and read their bra per lane, so the
// register J/K kernel can pack the kets of several bra pairs into one warp.
constexpr int kKetOuterMaxLab = 2;

// Primitive pairs of one side of a quartet: record i at rec + i * stride.
// GLOBAL: in global memory (vector read-only loads); otherwise built on the
// fly by the caller.
template <typename T, bool GLOBAL>
struct PrimList {
  const typename RecType<T>::type* rec;
  int stride;
  int n;
  __device__ __forceinline__ typename RecType<T>::type get(int i) const {
    if constexpr (GLOBAL)
      return ld_rec(rec + i * stride);
    else
      return rec[i * stride];
  }
};

// The vectors between the centres of a quartet that its integrals depend on.
template <typename T>
struct QuartetGeom {
  Vec3<T> AB, CD, CA;  // B - A, D - C, A - C
};
// From absolute centres; the differences are taken in FP64.
template <typename T>
__device__ __forceinline__ QuartetGeom<T> quartet_geom(const double* A, const double* B, const double* C,
                                                       const double* D) {
  return QuartetGeom<T>{Vec3<T>{T(B[0] - A[0]), T(B[1] - A[1]), T(B[2] - A[2])},
                        Vec3<T>{T(D[0] - C[0]), T(D[1] - C[1]), T(D[2] - C[2])},
                        Vec3<T>{T(A[0] - C[0]), T(A[1] - C[1]), T(A[2] - C[2])}};
}

// Accumulates the contracted block (ab|cd) for the ket Cartesian pairs of
// part PART into out[ab][cdi] (cd = CD0 + cdi).  Loops over all primitive
// pairs of the bra (outer) and ket (inner) shell pairs.  The bra E
// coefficients live in `ebra` (3 axes); with SHARED_BRA the bra pair is the
// same for the whole warp, `ebra` is warp-private shared memory and lanes
// 0..2 fill one axis each (every lane of the warp must call this function).
template <typename T, int LA, int LB, int LC, int LD, int NS, int PART, bool SHARED_BRA, bool GLOBAL_PP = true>
__device__ __forceinline__ void quartet_accumulate(
    const PrimList<T, GLOBAL_PP>& bra, const PrimList<T, GLOBAL_PP>& ket, const QuartetGeom<T>& geo,
    const T* __restrict__ boys_tab, T (*ebra)[LA + 1][LB + 1][LA + LB + 1],
    T (&out)[QCfg<LA, LB, LC, LD, NS, PART>::NAB][QCfg<LA, LB, LC, LD, NS, PART>::CDP]) {
  using Cfg = QCfg<LA, LB, LC, LD, NS, PART>;
  constexpr int L = Cfg::L;
  constexpr int LAB = Cfg::LAB;
  static_for<Cfg::NAB>([&](auto ab) {
    static_for<Cfg::CDP>([&](auto c) { out[decltype(ab)::value][decltype(c)::value] = T(0); });
  });
  if constexpr (Cfg::NCDP > 0) {
    using Rec = typename RecType<T>::type;
    // One primitive quartet: R, stage 1 (ket E against R) and stage 2 (bra E).
    auto prim = [&](const Rec& bp, const EArr<T, LA, LB> Ex, const EArr<T, LA, LB> Ey, const EArr<T, LA, LB> Ez,
                    const Rec& kp, const EArr<T, LC, LD> Fx, const EArr<T, LC, LD> Fy, const EArr<T, LC, LD> Fz,
                    const Vec3<T>& PQ) {
      T R[nherm(L)];
      prim_quartet_R<T, L>(bp.p, kp.p, bp.W * kp.W, PQ.x, PQ.y, PQ.z, boys_tab, R);
      static_for<Cfg::NCDP>([&](auto cdi_) {
        constexpr int cdi = decltype(cdi_)::value;
        constexpr int cd = Cfg::CD0 + cdi, c = cd / Cfg::ND, d = cd % Cfg::ND;
        constexpr int cx = cart_lx(LC, c), cy = cart_ly(LC, c), cz = cart_lz(LC, c);
        constexpr int dx = cart_lx(LD, d), dy = cart_ly(LD, d), dz = cart_lz(LD, d);
        // stage 1: X_tuv = sum_{t'u'v'} F^x F^y F^z R_{t+t',u+u',v+v'}
        T X[nherm(LAB)];
        static_for<nherm(LAB)>([&](auto h) { X[decltype(h)::value] = T(0); });
        static_for<cx + dx + 1>([&](auto tp_) {
          constexpr int tp = decltype(tp_)::value;
          static_for<cy + dy + 1>([&](auto up_) {
            constexpr int up = decltype(up_)::value;
            const T fxy = Fx[cx][dx][tp] * Fy[cy][dy][up];
            static_for<cz + dz + 1>([&](auto vp_) {
              constexpr int vp = decltype(vp_)::value;
              const T f = fxy * Fz[cz][dz][vp];
              static_for<nherm(LAB)>([&](auto h_) {
                constexpr int h = decltype(h_)::value;
                constexpr int s = (h >= 20) ? 4 : (h >= 10) ? 3 : (h >= 4) ? 2 : (h >= 1) ? 1 : 0;
                constexpr int k = h - s * (s + 1) * (s + 2) / 6;
                constexpr int t = cart_lx(s, k), u = cart_ly(s, k), v = s - t - u;
                X[h] += f * R[herm_index(t + tp, u + up, v + vp)];
              });
            });
          });
        });
        // stage 2: out[ab][cd] += sum_tuv E^x E^y E^z X_tuv
        static_for<Cfg::NA>([&](auto a_) {
          constexpr int a = decltype(a_)::value;
          constexpr int ax = cart_lx(LA, a), ay = cart_ly(LA, a), az = cart_lz(LA, a);
          static_for<Cfg::NB>([&](auto b_) {
            constexpr int b = decltype(b_)::value;
            constexpr int bx = cart_lx(LB, b), by = cart_ly(LB, b), bz = cart_lz(LB, b);
            T acc = T(0);
            static_for<ax + bx + 1>([&](auto t_) {
              constexpr int t = decltype(t_)::value;
              static_for<ay + by + 1>([&](auto u_) {
                constexpr int u = decltype(u_)::value;
                const T exy = Ex[ax][bx][t] * Ey[ay][by][u];
                static_for<az + bz + 1>([&](auto v_) {
                  constexpr int v = decltype(v_)::value;
                  acc += exy * Ez[az][bz][v] * X[herm_index(t, u, v)];
                });
              });
            });
            out[a * Cfg::NB + b][cdi] += acc;
          });
        });
      });
    };
    auto ket_e = [&](const Rec& kp, T (*fbuf)[LC + 1][LD + 1][LC + LD + 1]) {
      ecoef_compute<T, LC, LD, true>(fbuf[0], kp.t * geo.CD.x, kp.t * geo.CD.x - geo.CD.x, kp.h);
      ecoef_compute<T, LC, LD, true>(fbuf[1], kp.t * geo.CD.y, kp.t * geo.CD.y - geo.CD.y, kp.h);
      ecoef_compute<T, LC, LD, true>(fbuf[2], kp.t * geo.CD.z, kp.t * geo.CD.z - geo.CD.z, kp.h);
    };
    auto bra_e = [&](const Rec& bp, T ab, EArr<T, LA, LB> e) {
      ecoef_compute<T, LA, LB, false>(e, bp.t * ab, bp.t * ab - ab, bp.h);
    };
    if constexpr (GLOBAL_PP && LA + LB <= kKetOuterMaxLab) {
      // Ket primitives outer: each lane reads its ket primitive pair and its
      // E coefficients once; the bra primitive pairs (the same address in
      // every lane: one broadcast read) and their few E coefficients are
      // redone per ket primitive in registers.  Cuts the per-lane global
      // reads of the low-L classes, which are bound by L1 throughput.
      for (int iq = 0; iq < ket.n; ++iq) {
        const Rec kp = ket.get(iq);
        T fbuf[3][LC + 1][LD + 1][LC + LD + 1];
        ket_e(kp, fbuf);
        // A - Q
        const Vec3<T> AQ{geo.CA.x - kp.t * geo.CD.x, geo.CA.y - kp.t * geo.CD.y, geo.CA.z - kp.t * geo.CD.z};
        for (int ip = 0; ip < bra.n; ++ip) {
          const Rec bp = bra.get(ip);
          T eb[3][LA + 1][LB + 1][LA + LB + 1];
          bra_e(bp, geo.AB.x, eb[0]);
          bra_e(bp, geo.AB.y, eb[1]);
          bra_e(bp, geo.AB.z, eb[2]);
          const Vec3<T> PQ{AQ.x + bp.t * geo.AB.x, AQ.y + bp.t * geo.AB.y, AQ.z + bp.t * geo.AB.z};
          prim(bp, eb[0], eb[1], eb[2], kp, fbuf[0], fbuf[1], fbuf[2], PQ);
        }
      }
    } else {
      const int lane = threadIdx.x & 31;
      for (int ip = 0; ip < bra.n; ++ip) {
        const Rec bp = bra.get(ip);
        if constexpr (SHARED_BRA) {
          __syncwarp();
          if (lane == 0) bra_e(bp, geo.AB.x, ebra[0]);
          if (lane == 1) bra_e(bp, geo.AB.y, ebra[1]);
          if (lane == 2) bra_e(bp, geo.AB.z, ebra[2]);
          __syncwarp();
        } else {
          bra_e(bp, geo.AB.x, ebra[0]);
          bra_e(bp, geo.AB.y, ebra[1]);
          bra_e(bp, geo.AB.z, ebra[2]);
        }
        // P - C
        const Vec3<T> PC{geo.CA.x + bp.t * geo.AB.x, geo.CA.y + bp.t * geo.AB.y, geo.CA.z + bp.t * geo.AB.z};
        for (int iq = 0; iq < ket.n; ++iq) {
          const Rec kp = ket.get(iq);
          T fbuf[3][LC + 1][LD + 1][LC + LD + 1];
          ket_e(kp, fbuf);
          const Vec3<T> PQ{PC.x - kp.t * geo.CD.x, PC.y - kp.t * geo.CD.y, PC.z - kp.t * geo.CD.z};
          prim(bp, ebra[0], ebra[1], ebra[2], kp, fbuf[0], fbuf[1], fbuf[2], PQ);
        }
      }
    }
  }
}

// Dispatch a runtime part index (uniform over the block: blockIdx.y) to the
// compile-time PART of a functor template.
#define JQC_PART_CASE(P)                                    \
  case P:                                                   \
    if constexpr (P < NS) f.template run<P>();             \
    break;
template <int NS, typename F>
__device__ __forceinline__ void dispatch_part(int part, F& f) {
  switch (part) {
    JQC_PART_CASE(0) JQC_PART_CASE(1) JQC_PART_CASE(2) JQC_PART_CASE(3)
    JQC_PART_CASE(4) JQC_PART_CASE(5) JQC_PART_CASE(6) JQC_PART_CASE(7)
    JQC_PART_CASE(8) JQC_PART_CASE(9) JQC_PART_CASE(10) JQC_PART_CASE(11)
    JQC_PART_CASE(12) JQC_PART_CASE(13) JQC_PART_CASE(14) JQC_PART_CASE(15)
    default: break;
  }
}
#undef JQC_PART_CASE

// Number of parts the ket Cartesian pairs of a class are split into, so that
// one thread holds at most ~40 accumulators.
__host__ __device__ constexpr int class_split(int la, int lb, int lc, int ld) {
  int nab = ncart(la) * ncart(lb), ncd = ncart(lc) * ncart(ld);
  int ns = 1;
  while (ns < 16 && nab * ((ncd + ns - 1) / ns) > 40 && ns < ncd) ns *= 2;
  return ns;
}

}  // namespace jqc
