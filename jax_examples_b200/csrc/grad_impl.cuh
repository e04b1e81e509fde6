// Register-path ERI-derivative adjoint kernel (lane = ket pair).
//
// Work mapping of the J/K kernels: one warp per bra pair and up to 32 ket
// pairs, one lane per shell quartet, blockIdx.y selecting the part of the ket
// Cartesian pairs a thread handles.
//
// Gamma is contracted with the bra's E coefficients before any integral is
// formed.  With I = sum_abcd Gamma_abcd (ab|cd) of one primitive quartet,
// E^{ab}_h = K e^{ab}_h(P-A, P-B, p) and the property d e^{ij}_t / d(P-A) =
// i e^{i-1,j}_t (likewise with j for P-B), the force on the bra's centres is
//   dI/dA = (alpha/p) dI/dP - 2 mu (A-B) I + M     mu = alpha beta / p
//   dI/dB = (beta/p)  dI/dP + 2 mu (A-B) I - M
//   M_x   = sum Gamma [ -(beta/p) i e^{i-1,j} + (alpha/p) j e^{i,j-1} ] ...
// and the ket's likewise with dI/dQ = -dI/dP, so a primitive quartet needs the
// scalar I and three vectors.  Per bra primitive pair each lane forms, for
// its cd, the Hermite vectors
//   H[h]   = sum_ab Gamma_abcd e^{ab}_h         HM_x[h] = the same with M_x
// and per ket primitive pair, streaming over the bra Hermite index with
// X[h] = sum_k e^{cd}_k R_{h+k} (never stored),
//   I += H[h] X[h], dI/dP_x += H[h-1_x] X[h], M_x += HM_x[h] X[h],
//   N_x += H[h] sum_k n^{cd,x}_k R_{h+k}        (the ket's M)
// The earlier form built the derivative integrals of every ab with raised and
// lowered E coefficients and contracted them with Gamma afterwards: five times
// the arithmetic for a d-shell bra, 36 unrolled derivative blocks in (dd|ss).
// (H2O)16 6-31G*, screened at 1e-9, us: (dd|ss) 1646 -> 131, (dp|ss) 951 -> 223,
// (dp|ps) 1602 -> 442, (pp|ps) 1107 -> 276, (pp|ss) 633 -> 235, (ps|ss) 1100 ->
// 792; with (dd|ps) 1423 -> 249, (dp|ds) 1455 -> 462 and (dp|pp) 969 -> 384,
// which the row engine had, the classes' sum 18.1 -> 7.0 ms.  Bound by FP64
// latency at 8 warps a multiprocessor (255 registers).
#pragma once

#include "jk_impl.cuh"

namespace jqc {

// Doubles a lane may hold for Gamma, H, HM of its ket Cartesian pairs and R
// before the pairs are split over more block parts (each part evaluates R
// again): beyond the 127 that fit in registers, but the spills of a little
// more cost less than another R.  (H2O)16 screened / (H2O)5 gradient, ms: 80
// 10.9 / 2.06, 100 10.6 / 2.05, 128 10.2 / 2.12, 160 10.1 / 2.18, 200 10.1 / 2.23.
constexpr int kGradLaneDoubles = 128;

__host__ __device__ constexpr int grad_split(int la, int lb, int lc, int ld) {
  const int nab = ncart(la) * ncart(lb), ncd = ncart(lc) * ncart(ld), lab = la + lb;
  const int per = nab + nherm(lab) + (lab > 0 ? 3 * nherm(lab - 1) : 0);
  int cdp = ncd;
  while (cdp > 1 && cdp * per + nherm(lab + lc + ld + 1) > kGradLaneDoubles) --cdp;
  while ((ncd + cdp - 1) / cdp > 16) ++cdp;
  return (ncd + cdp - 1) / cdp;
}

// e^{ij}_t of the three axes and the coefficients of M.
template <int LA, int LB>
struct GradBraSmem {
  static constexpr int LAB = LA + LB;
  double E[3][LA + 1][LB + 1][LAB + 1];
  double M[3][LA + 1][LB + 1][LAB > 0 ? LAB : 1];  // t <= i + j - 1
};

// Decode compile-time Hermite index h into (t,u,v).
template <int H>
struct HermDecode {
  static constexpr int s = (H >= 84) ? 7 : (H >= 56) ? 6 : (H >= 35) ? 5 : (H >= 20) ? 4 : (H >= 10) ? 3 : (H >= 4) ? 2 : (H >= 1) ? 1 : 0;
  static constexpr int k = H - s * (s + 1) * (s + 2) / 6;
  static constexpr int t = cart_lx(s, k), u = cart_ly(s, k), v = s - t - u;
};

// m[i][j][t] = wj j e^{i,j-1}_t - wi i e^{i-1,j}_t
template <int LI, int LJ>
__device__ __forceinline__ void grad_m_coef(double (*m)[LJ + 1][LI + LJ > 0 ? LI + LJ : 1],
                                            const double (*e)[LJ + 1][LI + LJ + 1], double wi, double wj) {
  static_for<LI + 1>([&](auto i_) {
    static_for<LJ + 1>([&](auto j_) {
      constexpr int i = decltype(i_)::value, j = decltype(j_)::value;
      static_for<i + j>([&](auto t_) {
        constexpr int t = decltype(t_)::value;
        double v = 0.0;
        if constexpr (j > 0) v += (wj * j) * e[i][j - 1][t];
        if constexpr (i > 0) v -= (wi * i) * e[i - 1][j][t];
        m[i][j][t] = v;
      });
    });
  });
}

template <int LA, int LB, int LC, int LD, int NS>
struct GradBody {
  const GradParams& prm;
  int warp, lane;
  GradBraSmem<LA, LB>* sb;

  template <int PART>
  __device__ __forceinline__ void run() {
    using Cfg = QCfg<LA, LB, LC, LD, NS, PART>;
    if constexpr (Cfg::NCDP > 0) body<PART>();
  }

  template <int PART>
  __device__ __forceinline__ void body() {
    using Cfg = QCfg<LA, LB, LC, LD, NS, PART>;
    constexpr int NA = Cfg::NA, NB = Cfg::NB, ND = Cfg::ND;
    constexpr int NCDP = Cfg::NCDP;
    constexpr int L = Cfg::L, LAB = Cfg::LAB;
    constexpr int NH0 = nherm(LAB), NH1 = nherm(LAB + 1), NHM = LAB > 0 ? nherm(LAB - 1) : 0;

    const Task task = prm.tasks[warp];
    const ShellPair bp = prm.pairs[task.bra];
    const bool in_range = lane < int(task.nket);
    const int kidx = task.ket0 + (in_range ? lane : 0);
    const ShellPair kp = prm.pairs[kidx];
    bool active = in_range;
    if (prm.dmax_top != nullptr && active &&
        float(bp.Q) * float(kp.Q) * gamma_bound_top(prm, *prm.dmax_top) < prm.dens_tau)
      active = false;  // below the bound for any density block: no gathers
    if (prm.dmax != nullptr && active &&
        float(bp.Q) * float(kp.Q) * gamma_bound(prm, bp.a, bp.b, kp.a, kp.b) < prm.dens_tau)
      active = false;
    if (__ballot_sync(0xffffffffu, active) == 0u) return;
    const double* ctr = prm.centres;
    const Vec3<double> A{ctr[3 * bp.a], ctr[3 * bp.a + 1], ctr[3 * bp.a + 2]};
    const Vec3<double> B{ctr[3 * bp.b], ctr[3 * bp.b + 1], ctr[3 * bp.b + 2]};
    const Vec3<double> C{ctr[3 * kp.a], ctr[3 * kp.a + 1], ctr[3 * kp.a + 2]};
    const Vec3<double> Dc{ctr[3 * kp.b], ctr[3 * kp.b + 1], ctr[3 * kp.b + 2]};
    const int n = prm.n;
    const int a0 = prm.ao[bp.a], b0 = prm.ao[bp.b], c0 = prm.ao[kp.a], d0 = prm.ao[kp.b];

    // Gamma for this thread's part
    double G[Cfg::NAB][Cfg::CDP];
    static_for<Cfg::NAB * NCDP>([&](auto x_) {
      constexpr int x = decltype(x_)::value;
      constexpr int ab = x / NCDP, cdi = x % NCDP, cd = Cfg::CD0 + cdi;
      const int ia = a0 + ab / NB, ib = b0 + ab % NB, ic = c0 + cd / ND, id = d0 + cd % ND;
      double dab = 0.0, dcd = 0.0, kx = 0.0;
      if (active) {
        for (int s = 0; s < prm.n_dens; ++s) {
          const double* Ds = prm.D + (size_t)s * n * n;
          dab += __ldg(Ds + (size_t)ia * n + ib);
          dcd += __ldg(Ds + (size_t)ic * n + id);
          kx += __ldg(Ds + (size_t)ia * n + ic) * __ldg(Ds + (size_t)ib * n + id) +
                __ldg(Ds + (size_t)ia * n + id) * __ldg(Ds + (size_t)ib * n + ic);
        }
      }
      G[ab][cdi] = prm.jscale * dab * dcd - 0.5 * prm.kscale * kx;
    });
    // forces on A, on A + B (= dI/dP) and on C; D follows from translation
    double gA[3] = {0, 0, 0}, gP[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
    const int k0 = task.ket_begin(), k1 = active ? task.ket_end(kp.npp) : k0;  // ket primitive-pair range

    const int p0 = task.flags & 0xffff, p1 = task.flags >> 16;  // bra primitive-pair range
    for (int ip = p0; ip < p1; ++ip) {
      const PrimPair bpp = ld_pp(prm.pp + bp.pp + ip);
      const double wa = 2.0 * bpp.alpha * bpp.h, wb = 2.0 * bpp.beta * bpp.h;  // alpha / p, beta / p
      __syncwarp();
      if (lane < 3) {
        const double P = lane == 0 ? bpp.Px : lane == 1 ? bpp.Py : bpp.Pz;
        const double a = lane == 0 ? A.x : lane == 1 ? A.y : A.z;
        const double b = lane == 0 ? B.x : lane == 1 ? B.y : B.z;
        ecoef_compute<double, LA, LB, false>(sb->E[lane], P - a, P - b, bpp.h);
        grad_m_coef<LA, LB>(sb->M[lane], sb->E[lane], wb, wa);
      }
      __syncwarp();
      double H[Cfg::CDP][NH0], HM[Cfg::CDP][3][NHM > 0 ? NHM : 1];
      static_for<NCDP>([&](auto cdi_) {
        constexpr int cdi = decltype(cdi_)::value;
        static_for<NH0>([&](auto h_) { H[cdi][decltype(h_)::value] = 0.0; });
        static_for<NHM>([&](auto h_) {
          constexpr int h = decltype(h_)::value;
          HM[cdi][0][h] = HM[cdi][1][h] = HM[cdi][2][h] = 0.0;
        });
      });
      static_for<NA * NB>([&](auto ab_) {
        constexpr int ab = decltype(ab_)::value, ia = ab / NB, ib = ab % NB;
        constexpr int ax = cart_lx(LA, ia), ay = cart_ly(LA, ia), az = cart_lz(LA, ia);
        constexpr int bx = cart_lx(LB, ib), by = cart_ly(LB, ib), bz = cart_lz(LB, ib);
        static_for<ax + bx + 1>([&](auto t_) {
          constexpr int t = decltype(t_)::value;
          static_for<ay + by + 1>([&](auto u_) {
            constexpr int u = decltype(u_)::value;
            static_for<az + bz + 1>([&](auto v_) {
              constexpr int v = decltype(v_)::value;
              const double ex = sb->E[0][ax][bx][t], ey = sb->E[1][ay][by][u], ez = sb->E[2][az][bz][v];
              const double e = ex * ey * ez;
              static_for<NCDP>([&](auto c_) { H[decltype(c_)::value][herm_index(t, u, v)] += G[ab][decltype(c_)::value] * e; });
              if constexpr (t < ax + bx) {
                const double m = sb->M[0][ax][bx][t] * ey * ez;
                static_for<NCDP>([&](auto c_) { HM[decltype(c_)::value][0][herm_index(t, u, v)] += G[ab][decltype(c_)::value] * m; });
              }
              if constexpr (u < ay + by) {
                const double m = ex * sb->M[1][ay][by][u] * ez;
                static_for<NCDP>([&](auto c_) { HM[decltype(c_)::value][1][herm_index(t, u, v)] += G[ab][decltype(c_)::value] * m; });
              }
              if constexpr (v < az + bz) {
                const double m = ex * ey * sb->M[2][az][bz][v];
                static_for<NCDP>([&](auto c_) { HM[decltype(c_)::value][2][herm_index(t, u, v)] += G[ab][decltype(c_)::value] * m; });
              }
            });
          });
        });
      });
      double sI = 0.0, sP[3] = {0, 0, 0}, sM[3] = {0, 0, 0};  // over the ket primitives
      for (int iq = k0; iq < k1; ++iq) {
        const PrimPair kpp = ld_pp(prm.pp + kp.pp + iq);
        const double wc = 2.0 * kpp.alpha * kpp.h, wd = 2.0 * kpp.beta * kpp.h;
        double F[3][LC + 1][LD + 1][LC + LD + 1], N[3][LC + 1][LD + 1][LC + LD > 0 ? LC + LD : 1];
        ecoef_compute<double, LC, LD, true>(F[0], kpp.Px - C.x, kpp.Px - Dc.x, kpp.h);
        ecoef_compute<double, LC, LD, true>(F[1], kpp.Py - C.y, kpp.Py - Dc.y, kpp.h);
        ecoef_compute<double, LC, LD, true>(F[2], kpp.Pz - C.z, kpp.Pz - Dc.z, kpp.h);
        static_for<3>([&](auto x_) { grad_m_coef<LC, LD>(N[decltype(x_)::value], F[decltype(x_)::value], wd, wc); });
        double R[nherm(L + 1)];
        prim_quartet_R<double, L + 1>(bpp, kpp, prm.boys_al, R);
        double I = 0.0, dP[3] = {0, 0, 0}, n3[3] = {0, 0, 0};
        static_for<NCDP>([&](auto cdi_) {
          constexpr int cdi = decltype(cdi_)::value;
          constexpr int cd = Cfg::CD0 + cdi, c = cd / ND, d = cd % ND;
          constexpr int cx = cart_lx(LC, c), cy = cart_ly(LC, c), cz = cart_lz(LC, c);
          constexpr int dx = cart_lx(LD, d), dy = cart_ly(LD, d), dz = cart_lz(LD, d);
          constexpr int KX = cx + dx, KY = cy + dy, KZ = cz + dz;
          // products of the ket coefficients for this cd
          double fk[KX + 1][KY + 1][KZ + 1];
          static_for<KX + 1>([&](auto t_) {
            constexpr int t = decltype(t_)::value;
            static_for<KY + 1>([&](auto u_) {
              constexpr int u = decltype(u_)::value;
              const double fxy = F[0][cx][dx][t] * F[1][cy][dy][u];
              static_for<KZ + 1>([&](auto v_) { fk[t][u][decltype(v_)::value] = fxy * F[2][cz][dz][decltype(v_)::value]; });
            });
          });
          static_for<NH1>([&](auto h_) {
            constexpr int h = decltype(h_)::value;
            using Hd = HermDecode<h>;
            double X = 0.0;
            static_for<KX + 1>([&](auto t_) {
              static_for<KY + 1>([&](auto u_) {
                static_for<KZ + 1>([&](auto v_) {
                  constexpr int t = decltype(t_)::value, u = decltype(u_)::value, v = decltype(v_)::value;
                  X += fk[t][u][v] * R[herm_index(Hd::t + t, Hd::u + u, Hd::v + v)];
                });
              });
            });
            if constexpr (h < NH0) I += H[cdi][h] * X;
            if constexpr (Hd::t > 0) dP[0] += H[cdi][herm_index(Hd::t > 0 ? Hd::t - 1 : 0, Hd::u, Hd::v)] * X;
            if constexpr (Hd::u > 0) dP[1] += H[cdi][herm_index(Hd::t, Hd::u > 0 ? Hd::u - 1 : 0, Hd::v)] * X;
            if constexpr (Hd::v > 0) dP[2] += H[cdi][herm_index(Hd::t, Hd::u, Hd::v > 0 ? Hd::v - 1 : 0)] * X;
            if constexpr (h < NHM) {
              sM[0] += HM[cdi][0][h] * X;
              sM[1] += HM[cdi][1][h] * X;
              sM[2] += HM[cdi][2][h] * X;
            }
            if constexpr (h < NH0) {
              // the ket's M, one axis at a time
              if constexpr (KX > 0) {
                double Y = 0.0;
                static_for<KX>([&](auto t_) {
                  static_for<KY + 1>([&](auto u_) {
                    static_for<KZ + 1>([&](auto v_) {
                      constexpr int t = decltype(t_)::value, u = decltype(u_)::value, v = decltype(v_)::value;
                      Y += N[0][cx][dx][t] * F[1][cy][dy][u] * F[2][cz][dz][v] *
                           R[herm_index(Hd::t + t, Hd::u + u, Hd::v + v)];
                    });
                  });
                });
                n3[0] += H[cdi][h] * Y;
              }
              if constexpr (KY > 0) {
                double Y = 0.0;
                static_for<KX + 1>([&](auto t_) {
                  static_for<KY>([&](auto u_) {
                    static_for<KZ + 1>([&](auto v_) {
                      constexpr int t = decltype(t_)::value, u = decltype(u_)::value, v = decltype(v_)::value;
                      Y += F[0][cx][dx][t] * N[1][cy][dy][u] * F[2][cz][dz][v] *
                           R[herm_index(Hd::t + t, Hd::u + u, Hd::v + v)];
                    });
                  });
                });
                n3[1] += H[cdi][h] * Y;
              }
              if constexpr (KZ > 0) {
                double Y = 0.0;
                static_for<KX + 1>([&](auto t_) {
                  static_for<KY + 1>([&](auto u_) {
                    static_for<KZ>([&](auto v_) {
                      constexpr int t = decltype(t_)::value, u = decltype(u_)::value, v = decltype(v_)::value;
                      Y += F[0][cx][dx][t] * F[1][cy][dy][u] * N[2][cz][dz][v] *
                           R[herm_index(Hd::t + t, Hd::u + u, Hd::v + v)];
                    });
                  });
                });
                n3[2] += H[cdi][h] * Y;
              }
            }
          });
        });
        sI += I;
        const double w2n = 2.0 * wc * kpp.beta;  // 2 nu
        gC[0] += n3[0] - wc * dP[0] - w2n * (C.x - Dc.x) * I;
        gC[1] += n3[1] - wc * dP[1] - w2n * (C.y - Dc.y) * I;
        gC[2] += n3[2] - wc * dP[2] - w2n * (C.z - Dc.z) * I;
        sP[0] += dP[0];
        sP[1] += dP[1];
        sP[2] += dP[2];
      }
      const double w2m = 2.0 * wa * bpp.beta;  // 2 mu
      gA[0] += sM[0] + wa * sP[0] - w2m * (A.x - B.x) * sI;
      gA[1] += sM[1] + wa * sP[1] - w2m * (A.y - B.y) * sI;
      gA[2] += sM[2] + wa * sP[2] - w2m * (A.z - B.z) * sI;
      gP[0] += sP[0];
      gP[1] += sP[1];
      gP[2] += sP[2];
    }
    // scatter: 4 s per canonical quartet; bra centres reduced over the warp
    double sc = active ? 4.0 : 0.0;
    if (bp.diag()) sc *= 0.5;
    if (kp.diag()) sc *= 0.5;
    if (task.bra == kidx) sc *= 0.5;
    double* pf = prm.pair_force;
    static_for<3>([&](auto k_) {
      constexpr int k = decltype(k_)::value;
      const double a = warp_sum(sc * gA[k]), p = warp_sum(sc * gP[k]);
      if (lane == 0) {
        atomicAdd(pf + 6 * task.bra + k, a);
        atomicAdd(pf + 6 * task.bra + 3 + k, p - a);
      }
    });
    // centre D by translational invariance
    if (active) {
      static_for<3>([&](auto k_) {
        constexpr int k = decltype(k_)::value;
        atomicAdd(pf + 6 * kidx + k, sc * gC[k]);
        atomicAdd(pf + 6 * kidx + 3 + k, -sc * (gP[k] + gC[k]));
      });
    }
  }
};

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) grad_kernel(const GradParams prm) {
  constexpr int NS = grad_split(LA, LB, LC, LD);
  __shared__ GradBraSmem<LA, LB> sB[4];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= prm.n_tasks) return;
  GradBody<LA, LB, LC, LD, NS> body{prm, warp, int(threadIdx.x & 31), &sB[threadIdx.x >> 5]};
  dispatch_part<NS>(blockIdx.y, body);
}

template <int LA, int LB, int LC, int LD>
cudaError_t launch_grad_class(const GradParams& p, cudaStream_t s) {
  constexpr int NS = grad_split(LA, LB, LC, LD);
  if (p.n_tasks == 0) return cudaSuccess;
  dim3 grid((p.n_tasks + 3) / 4, NS);
  grad_kernel<LA, LB, LC, LD><<<grid, 128, 0, s>>>(p);
  return cudaGetLastError();
}

// Classes whose gradient runs in the register kernels, by compilation unit.
// (dd|dp) and (dd|dd) were slower here (340 -> 431 and 108 -> 316 us: R to
// order 8 and 9 does not fit a lane) and keep the row engine.
#define JQC_FOR_GRAD_REG_SP(X) \
  X(0, 0, 0, 0, 0)             \
  X(1, 1, 0, 0, 0)             \
  X(2, 1, 0, 1, 0)             \
  X(3, 1, 1, 0, 0)             \
  X(4, 1, 1, 1, 0)             \
  X(5, 1, 1, 1, 1)
#define JQC_FOR_GRAD_REG_DS(X) \
  X(6, 2, 0, 0, 0)             \
  X(7, 2, 0, 1, 0)             \
  X(8, 2, 0, 1, 1)             \
  X(9, 2, 0, 2, 0)
#define JQC_FOR_GRAD_REG_DP(X) \
  X(10, 2, 1, 0, 0)            \
  X(11, 2, 1, 1, 0)
#define JQC_FOR_GRAD_REG_DD(X) \
  X(15, 2, 2, 0, 0)            \
  X(16, 2, 2, 1, 0)
#define JQC_FOR_GRAD_REG_DPPP(X) X(12, 2, 1, 1, 1)
#define JQC_FOR_GRAD_REG_DPDS(X) X(13, 2, 1, 2, 0)
#define JQC_FOR_GRAD_REG_DPDP(X) X(14, 2, 1, 2, 1)
#define JQC_FOR_GRAD_REG_DDPP(X) X(17, 2, 2, 1, 1)
#define JQC_FOR_GRAD_REG_DDDS(X) X(18, 2, 2, 2, 0)
cudaError_t launch_grad_reg_sp(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_ds(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_dp(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_dd(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_dppp(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_dpds(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_dpdp(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_ddpp(int qc, const GradParams& p, cudaStream_t s);
cudaError_t launch_grad_reg_ddds(int qc, const GradParams& p, cudaStream_t s);

}  // namespace jqc
