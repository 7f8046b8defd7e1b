// The Pi half of the right-hand side (src/evolution.jl:324-354) with its stencil inputs staged
// into shared memory by the Tensor Memory Accelerator: the B200 form of rhs_pi_kernel for
// blocks of N = 32 cells at q = 4.
//
// A persistent CTA of 12 warps works through tiles of the blocks: NP pairs of neighbouring points
// along x (the whole row) x TY rows x TZ planes. For each component v of a tile one thread issues two
// tiled tensor copies of the block's working array into shared memory, whole rows (x -4 .. 35):
//   h_v   the tile's rows and planes widened by SR = 2
//   Pi_v  widened by KR = 3 for the dissipation
// completing on an mbarrier; two such stages alternate, so that the copies of the next component (of
// the next tile after the last one) run while component v is computed. Each thread computes the two
// points (i0, i0 + 1), i0 = 0, 2, ..., from 16-byte shared loads: one load serves both points of
// every y and z tap and two x taps. A row's owned points start on a sector (row_lead), so the pairs'
// global loads and stores are 16 bytes too.
//
// The mixed derivatives are outer sums of inner sums: d_x d_y h = sum_a w_a D_y h(x + a), d_x d_z h and
// d_y d_z h outer sums of D_z h. An inner sum is formed once, by the thread that owns the pair (those
// beyond the tile by extra tasks), and read by the points around it from shared memory: 39 instead of 91
// FP64 operations a point and component, and 45 instead of 68 shared loads a pair, against forming them
// at each point. On 64 blocks a stage takes 520 to 614 us by stage (777 us with every inner sum formed where it is
// used and every copy of a shared point computed; 685 to 746 us the one-point kernel); it is bound by DRAM (2.35 to
// 2.8 GB, 4.4 TB/s) and by the latency of its shared loads at 12 warps an SM.
//
// The arithmetic is the one-point kernel's, operation for operation (the same stencil sums in
// the same order and the same contraction with the head's coefficients), so both kernels give
// the same bits.
//
// Waits on the mbarriers are bounded: a wait that gives up records TGH_ERR_TIMEOUT in the
// launch's status word, waits (bounded again) for the copies it issued to land, and the CTA
// returns without writing further; the next verb on the problem, or the one that waits for this launch, reads the
// word and refuses.
#pragma once
#include "rhs.cuh"
#include "tma.cuh"

namespace tgh {

namespace pitma {
constexpr int N1 = 33, G = 3, SR = 2, KR = 3;  // q = 4, N = 32
constexpr int XB = 40, XC = 4;                 // the boxes' rows, and the column of point i = 0
constexpr int THREADS = 384;
// one tile shape: pairs along x, rows, planes; its boxes and inner-sum arrays in doubles
template <int NP_, int TY_, int TZ_> struct Shape {
  static constexpr int NP = NP_, TY = TY_, TZ = TZ_, ROWS = TY * TZ;
  static constexpr int HY = TY + 2 * SR, HZ = TZ + 2 * SR, PY = TY + 2 * KR, PZ = TZ + 2 * KR;
  static constexpr int HN = XB * HY * HZ, PN = XB * PY * PZ;
  static constexpr int DY = TY + 2 * SR;                        // rows of D_z per plane
  static constexpr int DN = XB * ROWS + XB * DY * TZ;           // D_y, then D_z
  static constexpr int NE = 4 * ROWS + 2 * SR * TZ * NP;        // inner-sum pairs beyond the tile's own
  static_assert(NP * ROWS <= THREADS && NE <= THREADS, "a thread per pair and per extra inner sum");
  static_assert(HN * 8 % 128 == 0, "the copies land on 128-byte boundaries");
};
// blocks computed to 33 points along x or y: 17 pairs a row, 33 = 3 x 11 rows, 17 x 2 planes (the last one past
// the block)
using Whole = Shape<17, 11, 2>;
// blocks that leave their upper x and y faces to their neighbours: 16 pairs a row (a warp's rows share no bank,
// whatever the pitch), 32 = 4 x 8 rows, 11 x 3 planes of 32 or 33
using Inner = Shape<16, 8, 3>;
enum { SHAPE_WHOLE = 0, SHAPE_INNER = 1 };
constexpr int STAGE = (Whole::HN + Whole::PN) * 8;
constexpr int DBYTES = Inner::DN * 8;
constexpr int SMEM = 2 * STAGE + DBYTES + 16 + 128;             // two stages, inner sums, mbarriers, alignment
static_assert(STAGE % 128 == 0 && Inner::HN + Inner::PN <= Whole::HN + Whole::PN && Whole::DN <= Inner::DN,
              "the shared arrays hold either shape");
static_assert(SMEM <= 227 * 1024, "two stages fit in shared memory");
constexpr int TILESY = N1 / Whole::TY, TILESZ = (N1 + Whole::TZ - 1) / Whole::TZ;
constexpr int TILES = TILESY * TILESZ;                          // 3 x 17 = 51 per block
}  // namespace pitma

// issue component v's two boxes for tile (b, y0, z0) into the stage at s
template <class Sh>
__device__ __forceinline__ void pitma_issue(const PiMaps& M, unsigned s, unsigned bar, int b, int v, int y0, int z0) {
  using namespace pitma;
  mbar_expect_tx(bar, (Sh::HN + Sh::PN) * 8);
  // h: rows y0 + G - SR .., planes z0 + G - SR ..; Pi: widened by KR
  tma_load_4d(s, &M.h, 0, y0 + G - SR, z0 + G - SR, b * NV + v, bar);
  tma_load_4d(s + Sh::HN * 8, &M.pi, 0, y0 + G - KR, z0 + G - KR, b * NV + NC + v, bar);
}

__device__ __forceinline__ double2 lds2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ double2 ldg2(const double* p) { return *reinterpret_cast<const double2*>(p); }

// the inner sums of the mixed differences at the pair p along stride s (the reference's sum term by
// term, st_mixed_ref); r returns the four pairs read
__device__ __forceinline__ double2 inner_sum(const double* p, int s, double2 r[2 * pitma::SR]) {
  using namespace pitma;
  double2 in;
#pragma unroll
  for (int n = 0; n < 2 * SR; ++n) {
    const int e = n < SR ? n - SR : n - SR + 1;
    r[n] = lds2(p + e * s);
    const double t0 = __dmul_rn(d1s<4>(e), r[n].x), t1 = __dmul_rn(d1s<4>(e), r[n].y);
    in.x = n == 0 ? t0 : __dadd_rn(in.x, t0);
    in.y = n == 0 ? t1 : __dadd_rn(in.y, t1);
  }
  return in;
}
// first (paired, fused) and second (term by term) differences of the pair from its four neighbours and centre
__device__ __forceinline__ void pair_d1_d2(const double2 r[2 * pitma::SR], double2 c, double d1[2], double d2[2]) {
  using namespace pitma;
  d1[0] = d1[1] = 0.0;
#pragma unroll
  for (int k = 1; k <= SR; ++k) {
    d1[0] = fma(W<4>::d1(k), r[SR - 1 + k].x - r[SR - k].x, d1[0]);
    d1[1] = fma(W<4>::d1(k), r[SR - 1 + k].y - r[SR - k].y, d1[1]);
  }
  d2[0] = __dmul_rn(W<4>::d2(SR), r[0].x);
  d2[1] = __dmul_rn(W<4>::d2(SR), r[0].y);
#pragma unroll
  for (int k = -SR + 1; k <= SR; ++k) {
    const double2 u = k == 0 ? c : r[k < 0 ? k + SR : k + SR - 1];
    const double w = W<4>::d2(k < 0 ? -k : k);
    d2[0] = __dadd_rn(d2[0], __dmul_rn(w, u.x));
    d2[1] = __dadd_rn(d2[1], __dmul_rn(w, u.y));
  }
}
// outer sum over a row's x offsets of the inner sums around the pair at p (both points)
__device__ __forceinline__ void outer_x(const double* p, double out[2]) {
  using namespace pitma;
  double r[6];
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const double2 q = lds2(p - 2 + 2 * t);
    r[2 * t] = q.x;
    r[2 * t + 1] = q.y;
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    double o = __dmul_rn(d1s<4>(-SR), r[e]);
#pragma unroll
    for (int a = -SR + 1; a <= SR; ++a) {
      if (a == 0) continue;
      o = __dadd_rn(o, __dmul_rn(d1s<4>(a), r[2 + e + a]));
    }
    out[e] = o;
  }
}

// the CTA's view of its shared memory and of the copy it waits for next
struct PiCta {
  unsigned char* smem;
  double* D;            // the inner sums
  unsigned base, bar;   // shared addresses of the stages and of the two mbarriers
  int n;                // copies consumed: copy n is in stage n & 1, the mbarrier's phase n >> 1
};

// tile t of the launch: of the list in the batched form, the whole blocks from b0 on in the plain form
template <int MODE> __device__ __forceinline__ PiTile pitma_tile(const RhsArgs& A, int b0, int t) {
  using namespace pitma;
  if (MODE == MODE_STAGE) return A.ptiles[t];
  const int r = t % TILES;
  return PiTile{b0 + t / TILES, (unsigned char)(r % TILESY * Whole::TY), (unsigned char)(r / TILESY * Whole::TZ),
                SHAPE_WHOLE, 7};
}

// One tile: its ten components, each refilling the stage the one before has freed through issue(n + 1). False:
// a wait gave up.
template <class Sh, bool DISS, int MODE, class Issue>
__device__ __forceinline__ bool pitma_tile_body(const RhsArgs& A, const WaitStatus& stat, PiCta& cta, const PiTile T,
                                                Issue issue) {
  using namespace pitma;
  const int tid = threadIdx.x;
  unsigned char* smem = cta.smem;
  double* Dy = cta.D;
  double* Dz = Dy + XB * Sh::ROWS;
  // this thread's pair: points i0, i0 + 1 of row jj, plane kk
  const bool active = tid < Sh::NP * Sh::ROWS;
  const int i0 = 2 * (tid % Sh::NP), row = active ? tid / Sh::NP : 0;
  const int jj = row % Sh::TY, kk = row / Sh::TY;
  const int cH = i0 + XC + XB * ((jj + SR) + Sh::HY * (kk + SR));
  const int cP = i0 + XC + XB * ((jj + KR) + Sh::PY * (kk + KR));
  const int cDy = i0 + XC + XB * row;
  const int cDz = i0 + XC + XB * ((jj + SR) + Sh::DY * kk);
  constexpr int s3h = XB * Sh::HY, s3p = XB * Sh::PY;
  // the extra inner sum this thread forms: D_y, then D_z, one pair beyond each end of the tile's rows, and
  // D_z on the SR rows either side of the tile
  int eH = -1, eS = 0;
  double* eD = nullptr;
  if (tid < 4 * Sh::ROWS) {
    const int r = tid / 2 % Sh::ROWS, c = (tid & 1) ? XC + 2 * Sh::NP : XC - 2, j = r % Sh::TY, k = r / Sh::TY;
    const bool isy = tid < 2 * Sh::ROWS;
    eH = c + XB * ((j + SR) + Sh::HY * (k + SR));
    eS = isy ? XB : s3h;
    eD = isy ? Dy + c + XB * r : Dz + c + XB * ((j + SR) + Sh::DY * k);
  } else if (tid < Sh::NE) {
    const int n = tid - 4 * Sh::ROWS, c = XC + 2 * (n % Sh::NP), m = n / Sh::NP;
    const int jr = m % (2 * SR), k = m / (2 * SR), j = jr < SR ? jr : jr + Sh::TY;  // row j - SR of the tile
    eH = c + XB * (j + Sh::HY * (k + SR));
    eS = s3h;
    eD = Dz + c + XB * (j + Sh::DY * k);
  }

  constexpr int NX = point_pitch(N1), Wd = N1 + 2 * G, Wx = row_pitch(Wd, G);
  constexpr long S = (long)N1 * N1 * N1, SX = (long)NX * N1 * N1, sv = (long)Wx * Wd * Wd;
  static_assert(Wx == XB && row_lead(G) + G == XC, "the boxes are whole rows");
  const int b = T.b, j = T.y0 + jj, k = T.z0 + kk;
  // rows, planes and the second point of a pair past the block's computed box are computed and dropped
  const int ex = N1 - 1 + (T.full & 1), ey = N1 - 1 + ((T.full >> 1) & 1), ez = N1 - 1 + (T.full >> 2);
  const bool own0 = active && i0 < ex && j < ey && k < ez, own1 = own0 && i0 + 1 < ex;
  const int jc = j < N1 ? j : N1 - 1, kc = k < N1 ? k : N1 - 1;
  const long ic = i0 + (long)NX * (jc + (long)N1 * kc);
  const double* cf = A.coef + (long)b * SX + ic;
  const double2 ww = own0 ? ldg2(cf + CF_W * A.ncoef) : make_double2(-1.0, -1.0);
  const double w[2] = {ww.x, own1 ? ww.y : -1.0};
  const bool live[2] = {w[0] >= 0.0, w[1] >= 0.0};
  const bool any = live[0] || live[1], both = live[0] && live[1];
  double cb[2][14];
#pragma unroll
  for (int c = 0; c < 14; ++c) {
    const double2 q = any ? ldg2(cf + c * A.ncoef) : make_double2(0.0, 0.0);
    cb[0][c] = live[0] ? q.x : 0.0;
    cb[1][c] = live[1] ? q.y : 0.0;
  }
  const double ih = 1.0 / A.blk[8 * b + 3], ih2 = ih * ih;
  const long wo = (long)b * NV * sv + (i0 + G) + (long)Wx * ((jc + G) + (long)Wd * (kc + G));
  double* acc = MODE == MODE_STAGE ? A.acc + (long)b * NV * SX + ic : nullptr;
  double* du = MODE == MODE_DU ? A.du + (long)b * NV * S + i0 + N1 * (jc + (long)N1 * kc) : nullptr;

#pragma unroll 1
  for (int v = 0; v < NC; ++v, ++cta.n) {
    const int n = cta.n;
    // the epilogue's loads first: they are in flight while the copies land
    double2 m = make_double2(0, 0), kh = m, uh = m, up = m, ah = m, ap = m;
    if (any) {
      m = ldg2(cf + (CF_M0 + v) * A.ncoef);
      if (MODE == MODE_STAGE) {
        kh = ldg2(cf + (CF_DTH0 + v) * A.ncoef);
        if (A.stage != 4) {
          uh = ldg2(A.u0 + wo + v * sv);
          up = ldg2(A.u0 + wo + (NC + v) * sv);
        }
        if (A.stage != 1) {
          ah = ldg2(acc + v * SX);
          ap = ldg2(acc + (NC + v) * SX);
        }
      }
    }
    // every thread waits (bounded) for the stage; the CTA goes on only if all of them saw it.
    // The vote is also the barrier after the component before: its stage and the inner sums may
    // now be refilled.
    const bool got = mbar_wait(cta.bar + 8 * (n & 1), (n >> 1) & 1, stat.limit);
    if (!__syncthreads_and(got)) return false;
    if (tid == 0 && n >= 1) issue(n + 1);
    const double* H = reinterpret_cast<const double*>(smem + (n & 1) * STAGE);
    const double* P = H + Sh::HN;
    double s[2], p2[2], hd1[3][2], ko[2];
    // ---- h_v: the y and z taps give the inner sums and the y, z differences ----
    const double* hc = H + cH;
    {
      double hx[6];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const double2 r = lds2(hc - 2 + 2 * q);
        hx[2 * q] = r.x;
        hx[2 * q + 1] = r.y;
      }
      const double2 c = make_double2(hx[2], hx[3]);
      double2 r[2 * SR];
      double d2[2];
      const double2 iy = inner_sum(hc, XB, r);
      if (active) *reinterpret_cast<double2*>(Dy + cDy) = iy;
      pair_d1_d2(r, c, hd1[1], d2);
      p2[0] = d2[0];
      p2[1] = d2[1];
      const double2 iz = inner_sum(hc, s3h, r);
      if (active) *reinterpret_cast<double2*>(Dz + cDz) = iz;
      pair_d1_d2(r, c, hd1[2], d2);
      // x: first differences paired at +-k, second differences term by term
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double* u = hx + 2 + e;
        double a = 0.0;
#pragma unroll
        for (int kx = 1; kx <= SR; ++kx) a = fma(W<4>::d1(kx), u[kx] - u[-kx], a);
        hd1[0][e] = a;
        double d = __dmul_rn(W<4>::d2(SR), u[-SR]);
#pragma unroll
        for (int kx = -SR + 1; kx <= SR; ++kx) d = __dadd_rn(d, __dmul_rn(W<4>::d2(kx < 0 ? -kx : kx), u[kx]));
        double q = cb[e][CF_AXX] * d;
        q = fma(cb[e][CF_AYY], p2[e], q);
        p2[e] = fma(cb[e][CF_AZZ], d2[e], q);
      }
    }
    if (eH >= 0) {
      double2 r[2 * SR];
      *reinterpret_cast<double2*>(eD) = inner_sum(H + eH, eS, r);
    }
    // ---- Pi_v: x taps from five 16-byte loads, y and z taps one load an offset ----
    {
      const double* pc = P + cP;
      double px[10];
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        const double2 r = lds2(pc - 4 + 2 * q);
        px[2 * q] = r.x;
        px[2 * q + 1] = r.y;
      }
      double d1[3][2], kd[3][2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double* u = px + 4 + e;
        double a = 0.0;
#pragma unroll
        for (int kx = 1; kx <= SR; ++kx) a = fma(W<4>::d1(kx), u[kx] - u[-kx], a);
        d1[0][e] = a;
        double c = W<4>::ko(0) * u[0];
        kd[1][e] = kd[2][e] = c;
#pragma unroll
        for (int kx = 1; kx <= KR; ++kx) c = fma(W<4>::ko(kx), u[kx] + u[-kx], c);
        kd[0][e] = c;
      }
#pragma unroll
      for (int ax = 1; ax < 3; ++ax) {
        const int st = ax == 1 ? XB : s3p;
        d1[ax][0] = d1[ax][1] = 0.0;
#pragma unroll
        for (int kt = 1; kt <= KR; ++kt) {
          const double2 up2 = lds2(pc + kt * st), dn2 = lds2(pc - kt * st);
          if (kt <= SR) {
            d1[ax][0] = fma(W<4>::d1(kt), up2.x - dn2.x, d1[ax][0]);
            d1[ax][1] = fma(W<4>::d1(kt), up2.y - dn2.y, d1[ax][1]);
          }
          kd[ax][0] = fma(W<4>::ko(kt), up2.x + dn2.x, kd[ax][0]);
          kd[ax][1] = fma(W<4>::ko(kt), up2.y + dn2.y, kd[ax][1]);
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double* c = cb[e];
        double a = c[CF_B0] * (ih * d1[0][e]);
        a = fma(c[CF_B1], ih * d1[1][e], a);
        a = fma(c[CF_B2], ih * d1[2][e], a);
        a = fma(c[CF_DIVB], px[4 + e], a);
        a = fma(c[CF_DA0], ih * hd1[0][e], a);
        a = fma(c[CF_DA1], ih * hd1[1][e], a);
        s[e] = fma(c[CF_DA2], ih * hd1[2][e], a);
        ko[e] = kd[0][e] + kd[1][e] + kd[2][e];
      }
    }
    __syncthreads();  // the inner sums are written
    {
      double mxy[2], mxz[2], myz[2];
      outer_x(Dy + cDy, mxy);
      outer_x(Dz + cDz, mxz);
#pragma unroll
      for (int a = -SR; a <= SR; ++a) {
        if (a == 0) continue;
        const double2 q = lds2(Dz + cDz + a * XB);
        const double o0 = __dmul_rn(d1s<4>(a), q.x), o1 = __dmul_rn(d1s<4>(a), q.y);
        myz[0] = a == -SR ? o0 : __dadd_rn(myz[0], o0);
        myz[1] = a == -SR ? o1 : __dadd_rn(myz[1], o1);
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double* c = cb[e];
        double q = fma(c[CF_AXY], mxy[e], p2[e]);
        q = fma(c[CF_AXZ], mxz[e], q);
        q = fma(c[CF_AYZ], myz[e], q);
        s[e] = fma(ih2, q, s[e]);
        if (DISS) s[e] = fma(c[CF_EH], ko[e], s[e]);
      }
    }
    if (!any) continue;
    const double val0 = w[0] == 1.0 ? s[0] + m.x : fma(w[0], s[0], m.x);
    const double val1 = w[1] == 1.0 ? s[1] + m.y : fma(w[1], s[1], m.y);
    if (MODE == MODE_DU) {
      if (live[0]) du[(NC + v) * S] = val0;
      if (live[1]) du[(NC + v) * S + 1] = val1;
    } else {
      // the RK4 stage update of both halves of component v (EmitStage::fin)
      auto put = [&](double* p, double x, double y) {
        if (both) {
          *reinterpret_cast<double2*>(p) = make_double2(x, y);
        } else {
          if (live[0]) p[0] = x;
          if (live[1]) p[1] = y;
        }
      };
      double* nh = A.next + wo + v * sv;
      double* np = A.next + wo + (NC + v) * sv;
      if (A.stage == 4) {
        put(nh, fma(A.cb, kh.x, ah.x), fma(A.cb, kh.y, ah.y));
        put(np, fma(A.cb, val0, ap.x), fma(A.cb, val1, ap.y));
      } else {
        const bool first = A.stage == 1;
        put(acc + v * SX, fma(A.cb, kh.x, first ? uh.x : ah.x), fma(A.cb, kh.y, first ? uh.y : ah.y));
        put(acc + (NC + v) * SX, fma(A.cb, val0, first ? up.x : ap.x), fma(A.cb, val1, first ? up.y : ap.y));
        put(nh, fma(A.ca, kh.x, uh.x), fma(A.ca, kh.y, uh.y));
        put(np, fma(A.ca, val0, up.x), fma(A.ca, val1, up.y));
      }
    }
  }
  return true;
}

template <bool DISS, int MODE>
__global__ void __launch_bounds__(pitma::THREADS)
    rhs_pi_tma_kernel(const RhsArgs A, const __grid_constant__ TmaMaps M, const WaitStatus stat, int b0, int ntiles) {
  using namespace pitma;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  // the copies land on 128-byte boundaries
  const unsigned raw = smem_u32(smem_raw);
  const unsigned base = (raw + 127u) & ~127u;
  unsigned char* smem = smem_raw + (base - raw);
  PiCta cta{smem, reinterpret_cast<double*>(smem + 2 * STAGE), base, base + 2 * STAGE + DBYTES, 0};
  const int tid = threadIdx.x;
  // the CTA's tiles blockIdx.x, blockIdx.x + gridDim.x, ...; component v of its m-th tile is copy 10 m + v
  auto issue = [&](int n) {
    const int t = blockIdx.x + (n / NC) * gridDim.x;
    if (t >= ntiles) return;
    const PiTile T = pitma_tile<MODE>(A, b0, t);
    const unsigned s = base + (n & 1) * STAGE, bar = cta.bar + 8 * (n & 1);
    if (T.shape == SHAPE_INNER)
      pitma_issue<Inner>(M.inner, s, bar, T.b, n % NC, T.y0, T.z0);
    else
      pitma_issue<Whole>(M.whole, s, bar, T.b, n % NC, T.y0, T.z0);
  };
  if (tid == 0) {
    mbar_init(cta.bar, 1);
    mbar_init(cta.bar + 8, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    issue(0);
    issue(1);
  }
  __syncthreads();
  bool ok = true;
#pragma unroll 1
  for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x) {
    const PiTile T = pitma_tile<MODE>(A, b0, t);
    if (MODE == MODE_STAGE && T.shape == SHAPE_INNER)
      ok = pitma_tile_body<Inner, DISS, MODE>(A, stat, cta, T, issue);
    else
      ok = pitma_tile_body<Whole, DISS, MODE>(A, stat, cta, T, issue);
  }
  if (!ok) {
    // a wait gave up: record it, let the copies already issued (copy n, and copy 1 when n = 0)
    // land, bounded, then leave without writing further
    if (tid == 0) stat.gave_up();
    const long long drain = 1ll << 24;
    mbar_wait(cta.bar + 8 * (cta.n & 1), (cta.n >> 1) & 1, drain);
    if (cta.n == 0) mbar_wait(cta.bar + 8, 0, drain);
  }
}

}  // namespace tgh
