// Primitive blocks of the (dd|dp) and (dd|dd) classes (obara_saika.py:227-332
// primitive_eri_block with unit coefficients, K_AB and K_CD included).
//
// A block of kPrimHiThreads threads takes kPrimHiQuartets quartets through
// shared memory:
//   1. each warp builds E, the Boys values and R_tuv of its quartets, the
//      quartets' components side by side over the lanes;
//   2. thread (quartet, bra Hermite index h) reads R_{h+k} for every ket Hermite
//      index k and turns the ket side Cartesian: X[cd][h] for all cd;
//   3. thread (quartet, cd) reads its row X[cd][.] and turns the bra side
//      Cartesian in place;
//   4. the blocks are stored, consecutive threads on consecutive addresses.
// Both transformations go one axis at a time (hermite_to_cart), which uses each
// E coefficient for several sums: about 410 multiply-adds against 81
// coefficient reads a thread.  The column engine's form, used here before, did
// dense sums over the 35 x 35 Hermite pairs on 36 of 64 lane slots: 2^16 (dd|dd)
// quartets 982 -> 557 us.  Bound by latency: 12 warps a multiprocessor is what
// 14 KB of shared memory a quartet leaves room for (issue 37% of cycles, FP64
// pipe 23%, shared memory 66%).  Without the halves (6 warps, a quarter fewer
// instructions) 567 us; the R recursion with ten or sixteen lanes a quartet
// and its codes in registers 597 and 584 us.
#include "axis_transform.cuh"

namespace jqc {

constexpr int kPrimHiQuartets = 8;
// Two halves of 96 threads: 8 x 35 and 8 x 36 items fill 96 three times.  The
// halves share the items and take the Cartesian pairs with iz = 0 and iz > 0
// of each (18 of 36 outputs each for a dd pair): 12 instead of 6 warps a
// multiprocessor on the shared memory that limits the quartets in flight.
constexpr int kPrimHiHalf = 96;
constexpr int kPrimHiThreads = 2 * kPrimHiHalf;

template <int LA, int LB, int LC, int LD>
struct PrimHiQuartet {
  static constexpr int LAB = LA + LB, LCD = LC + LD, L = LAB + LCD;
  static constexpr int NAB = ncart(LA) * ncart(LB), NCD = ncart(LC) * ncart(LD);
  static constexpr int NHB = nherm(LAB);
  static constexpr int kRow = (NHB > NAB ? NHB : NAB) | 1;  // odd: rows on different banks
  double Eb[3][LA + 1][LB + 1][LAB + 1];
  double Ek[3][LC + 1][LD + 1][LCD + 1];  // with (-1)^t
  double R[nherm(L)];
  double X[NCD * kRow];  // P - Q and R^n_000 at first; X[cd][h]; then the block [cd][ab]
  __device__ __forceinline__ double* PQ() { return X; }
  __device__ __forceinline__ double* Rn() { return X + 3; }
};

template <int LA, int LB, int LC, int LD>
struct PrimHiSmem {
  using Q = PrimHiQuartet<LA, LB, LC, LD>;
  Q q[kPrimHiQuartets];
  int code[nherm(Q::L)];  // kRCode
  __align__(4) unsigned char sum[nherm(Q::LCD) * nherm(Q::LAB) + 3];  // kHermSum
};
// two blocks a multiprocessor: 228 KB, 1 KB of it the system's for each block
static_assert(2 * (sizeof(PrimHiSmem<2, 2, 2, 2>) + 1024) <= 228 * 1024, "only one block fits");

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(kPrimHiThreads, 2) prim_hi_kernel(const PrimQuartetParams prm) {
  using S = PrimHiSmem<LA, LB, LC, LD>;
  using Q = typename S::Q;
  constexpr int L = Q::L, LAB = Q::LAB, LCD = Q::LCD, NH = Q::NHB, NK = nherm(LCD), NCD = Q::NCD, NAB = Q::NAB;
  constexpr int kPer = 2;  // quartets a warp starts; the last warps have none
  static_assert(kPrimHiThreads / 32 * kPer >= kPrimHiQuartets, "too few warps");
  static_assert(nherm(L) <= 256 && kPer * 6 <= 32 && kPer * (L + 1) <= 32, "table or lane mapping too small");
  extern __shared__ __align__(16) unsigned char prim_hi_raw[];
  S& sm = *reinterpret_cast<S*>(prim_hi_raw);
  const int tid = int(threadIdx.x), lane = tid & 31, warp = tid >> 5;
  const long long q0 = (long long)blockIdx.x * kPrimHiQuartets;
  const int nq = (int)(prm.n - q0 < kPrimHiQuartets ? prm.n - q0 : kPrimHiQuartets);
  for (int i = tid; i < nherm(L); i += kPrimHiThreads) sm.code[i] = __ldg(kRCode.v + i);
  static_assert(NH == HermSumTable::N && NK <= HermSumTable::N, "the table is for a dd bra");
  for (int i = tid; i < (NK * NH + 3) / 4; i += kPrimHiThreads)
    reinterpret_cast<unsigned*>(sm.sum)[i] = __ldg(reinterpret_cast<const unsigned*>(kHermSum.v) + i);

  // 1. this warp's quartets [w0, w0 + wq)
  const int w0 = warp * kPer, wq = nq - w0 < kPer ? (nq > w0 ? nq - w0 : 0) : kPer;
  if (lane < wq * 6) {  // one axis of one side's E coefficients a lane
    const int ql = w0 + lane / 6, side = (lane % 6) / 3, ax = lane % 3;
    const double* ex = prm.exps + 4 * (q0 + ql) + 2 * side;
    const double* c = prm.centres + 12 * (q0 + ql) + 6 * side;
    const double al = ex[0], be = ex[1], p = al + be, P = (al * c[ax] + be * c[3 + ax]) / p;
    if (side == 0)
      ecoef_compute<double, LA, LB, false>(sm.q[ql].Eb[ax], P - c[ax], P - c[3 + ax], 0.5 / p);
    else
      ecoef_compute<double, LC, LD, true>(sm.q[ql].Ek[ax], P - c[ax], P - c[3 + ax], 0.5 / p);
  }
  if (lane < wq * (L + 1)) {  // one Boys order of one quartet a lane
    const int ql = w0 + lane / (L + 1), m = lane % (L + 1);
    const double* ex = prm.exps + 4 * (q0 + ql);
    const double* c = prm.centres + 12 * (q0 + ql);
    const double p = ex[0] + ex[1], q = ex[2] + ex[3];
    double r2 = 0.0, ab2 = 0.0, cd2 = 0.0, d[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const double ab = c[x] - c[3 + x], cd = c[6 + x] - c[9 + x];
      ab2 += ab * ab;
      cd2 += cd * cd;
      d[x] = (ex[0] * c[x] + ex[1] * c[3 + x]) / p - (ex[2] * c[6 + x] + ex[3] * c[9 + x]) / q;
      r2 += d[x] * d[x];
    }
    const double kab = exp(-(ex[0] * ex[1] / p) * ab2), kcd = exp(-(ex[2] * ex[3] / q) * cd2);
    const double r = rsqrt(p + q), rho = p * q * (r * r);
    double pref = kTwoPi25 * kab * kcd / (p * q) * r;
    for (int k = 0; k < m; ++k) pref *= -2.0 * rho;
    sm.q[ql].Rn()[m] = pref * boys_single<double>(rho * r2, m, prm.boys);
    if (m < 3) sm.q[ql].PQ()[m] = m == 0 ? d[0] : (m == 1 ? d[1] : d[2]);
  }
  __syncthreads();  // also publishes the tables
  if (lane < wq) sm.q[w0 + lane].R[0] = sm.q[w0 + lane].Rn()[L];
  __syncwarp();
  // R_tuv in place (warp_hermite_R), the warp's quartets side by side
  static_for<L>([&](auto i_) {
    constexpr int n = L - 1 - decltype(i_)::value;
    static_for<L - n>([&](auto j_) {
      constexpr int s = L - n - decltype(j_)::value;
#pragma unroll
      for (int b = 0; b < kPer * ncart(s); b += 32) {
        const int x = b + lane;
        if (x < wq * ncart(s)) {
          Q& q = sm.q[w0 + x / ncart(s)];
          const int k = x % ncart(s), c = sm.code[nherm(s - 1) + k];
          q.R[nherm(s - 1) + k] = q.PQ()[c >> 22] * q.R[c & 511] + double((c >> 18) & 15) * q.R[(c >> 9) & 511];
        }
      }
      __syncwarp();
    });
    if (lane < wq) sm.q[w0 + lane].R[0] = sm.q[w0 + lane].Rn()[n];
    __syncwarp();
  });
  __syncthreads();

  const int half = tid / kPrimHiHalf, ti = tid % kPrimHiHalf;  // half: uniform over a warp
  // 2. ket side
  for (int i = ti; i < nq * NH; i += kPrimHiHalf) {
    Q& q = sm.q[i / NH];
    const int h = i % NH;
    double r[NK];
    static_for<NK>([&](auto k_) {
      constexpr int k = decltype(k_)::value;
      r[k] = q.R[sm.sum[k * NH + h]];
    });
    auto put = [&](auto cd_, double v) { q.X[decltype(cd_)::value * Q::kRow + h] = v; };
    if (half == 0)
      hermite_to_cart<LC, LD, 0, 1>(r, q.Ek, put);
    else
      hermite_to_cart<LC, LD, 1, LC + 1>(r, q.Ek, put);
  }
  __syncthreads();
  // 3. bra side, in place: both threads of a row read it before either writes
  for (int b = 0; b < nq * NCD; b += kPrimHiHalf) {  // uniform over the block
    const int i = b + ti;
    const bool has = i < nq * NCD;
    Q& q = sm.q[has ? i / NCD : 0];
    double* row = q.X + (has ? i % NCD : 0) * Q::kRow;
    double x[NH];
    static_for<NH>([&](auto h_) { x[decltype(h_)::value] = row[decltype(h_)::value]; });
    __syncthreads();
    if (!has) continue;
    auto put = [&](auto ab_, double v) { row[decltype(ab_)::value] = v; };
    if (half == 0)
      hermite_to_cart<LA, LB, 0, 1>(x, q.Eb, put);
    else
      hermite_to_cart<LA, LB, 1, LA + 1>(x, q.Eb, put);
  }
  __syncthreads();
  // 4. two elements (ab, cd) and (ab, cd + 1) a thread; the pair index advances by
  // kPrimHiThreads = kStepAB * NCD / 2 + kStepCD (NCD is even, so every pair is
  // 16-byte aligned where the caller's array is)
  constexpr int NP = NCD / 2, kStepAB = kPrimHiThreads / NP, kStepCD = kPrimHiThreads % NP;
  static_assert(NCD % 2 == 0, "pairs of ket components");
  double* o = prm.out + q0 * (NAB * NCD);
  const bool wide = (reinterpret_cast<unsigned long long>(prm.out) & 15) == 0;
  for (int ql = 0; ql < nq; ++ql) {
    const double* x = sm.q[ql].X;
    int ab = tid / NP, cp = tid % NP;
    for (int e = tid; e < NAB * NP; e += kPrimHiThreads) {
      const double* v = x + 2 * cp * Q::kRow + ab;
      double* w = o + 2 * (ql * (NAB * NP) + e);
      if (wide) {
        *reinterpret_cast<double2*>(w) = make_double2(v[0], v[Q::kRow]);
      } else {
        w[0] = v[0];
        w[1] = v[Q::kRow];
      }
      ab += kStepAB;
      cp += kStepCD;
      if (cp >= NP) {
        cp -= NP;
        ++ab;
      }
    }
  }
}

template <int LA, int LB, int LC, int LD>
static cudaError_t launch_prim_hi_class(const PrimQuartetParams& p, cudaStream_t s) {
  constexpr int bytes = int(sizeof(PrimHiSmem<LA, LB, LC, LD>));
  cudaError_t e = cudaFuncSetAttribute(prim_hi_kernel<LA, LB, LC, LD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       bytes);
  if (e != cudaSuccess) return e;
  const long long blocks = (p.n + kPrimHiQuartets - 1) / kPrimHiQuartets;
  prim_hi_kernel<LA, LB, LC, LD><<<(unsigned)blocks, kPrimHiThreads, bytes, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_prim_hi(int qc, const PrimQuartetParams& p, cudaStream_t s) {
  switch (qc) {
    case 19:
      return launch_prim_hi_class<2, 2, 2, 1>(p, s);
    case 20:
      return launch_prim_hi_class<2, 2, 2, 2>(p, s);
    default:
      return cudaErrorNotSupported;
  }
}

}  // namespace jqc
