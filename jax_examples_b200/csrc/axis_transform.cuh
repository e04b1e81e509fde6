// Hermite to Cartesian transformation of one side of a quartet, one axis at a
// time, and the table of Hermite index sums: shared by the column engine and
// the high-L primitive blocks.
#pragma once

#include "warp_engine.cuh"

namespace jqc {

// val[ij] = sum_tuv e^x_t e^y_u e^z_v r[tuv] for every Cartesian pair of shells
// (LI, LJ) with iz in [IZ0, IZ1), z first: f(ij, val) with compile-time ij.
template <int LI, int LJ, int IZ0, int IZ1, typename T, typename F>
__device__ __forceinline__ void hermite_to_cart(const T (&r)[nherm(LI + LJ)],
                                                const T (*e)[LI + 1][LJ + 1][LI + LJ + 1], F&& f) {
  constexpr int L = LI + LJ;
  static_for<IZ1 - IZ0>([&](auto iz_) {
    static_for<LJ + 1>([&](auto jz_) {
      constexpr int iz = IZ0 + decltype(iz_)::value, jz = decltype(jz_)::value, TU = L - iz - jz;
      T y1[TU + 1][TU + 1];  // t + u <= TU
      static_for<TU + 1>([&](auto t_) {
        constexpr int t = decltype(t_)::value;
        static_for<TU + 1 - t>([&](auto u_) {
          constexpr int u = decltype(u_)::value;
          T s = T(0);
          static_for<iz + jz + 1>([&](auto v_) {
            constexpr int v = decltype(v_)::value;
            s += e[2][iz][jz][v] * r[herm_index(t, u, v)];
          });
          y1[t][u] = s;
        });
      });
      static_for<LI + 1 - iz>([&](auto iy_) {
        static_for<LJ + 1 - jz>([&](auto jy_) {
          constexpr int iy = decltype(iy_)::value, jy = decltype(jy_)::value;
          constexpr int ix = LI - iy - iz, jx = LJ - jy - jz;
          T val = T(0);
          static_for<ix + jx + 1>([&](auto t_) {
            constexpr int t = decltype(t_)::value;
            T s = T(0);
            static_for<iy + jy + 1>([&](auto u_) {
              constexpr int u = decltype(u_)::value;
              s += e[1][iy][jy][u] * y1[t][u];
            });
            val += e[0][ix][jx][t] * s;
          });
          // libint order: component (lx, ly, lz) of shell l at (l-lx)(l-lx+1)/2 + lz
          constexpr int i = (LI - ix) * (LI - ix + 1) / 2 + iz, j = (LJ - jx) * (LJ - jx + 1) / 2 + jz;
          f(std::integral_constant<int, i * ncart(LJ) + j>{}, val);
        });
      });
    });
  });
}

// Hermite index of h + k for h and k of total order <= 4, row k: built at
// compile time, copied to shared memory by every block.
struct HermSumTable {
  static constexpr int N = nherm(4);
  unsigned char v[N * N + 3];
  constexpr HermSumTable() : v() {
    for (int k = 0; k < N; ++k)
      for (int h = 0; h < N; ++h) {
        int s = 0, r = 0;
        while (nherm(s) <= h) ++s;
        while (nherm(r) <= k) ++r;
        const int a = s > 0 ? h - nherm(s - 1) : 0, b = r > 0 ? k - nherm(r - 1) : 0;
        v[k * N + h] = (unsigned char)herm_index(cart_lx(s, a) + cart_lx(r, b), cart_ly(s, a) + cart_ly(r, b),
                                                 cart_lz(s, a) + cart_lz(r, b));
      }
  }
};
__device__ constexpr __align__(4) HermSumTable kHermSum{};

}  // namespace jqc
