// The Pi half of the right-hand side from shared-memory tiles, for any block size and order in FP64:
// rhs_pi_tma_kernel's scheme (whole rows staged by the Tensor Memory Accelerator, two points along x a thread,
// every inner sum of the mixed differences formed once) with the tile's geometry chosen on the host for the
// block size, the order and the shared memory (pi_tile_geometry).
//
// The one-point kernel reads (2 R)^2 points through L1 for each of three mixed differences, 16 to 192 loads a
// component from q = 2 to 8, and is bound by their latency and wavefronts; here a point costs 8 R inner and outer
// terms. One right-hand side (head and Pi), 27 blocks of 27^3 at q = 8: 471 us (676 us with the one-point kernel);
// 64 of 24^3 at q = 6: 678 us (1,183), at q = 4: 536 us (779), at q = 2: 448 us (569).
//
// Where two stages of a component's boxes fit the shared memory the next component's copies run during the
// whole of this one; else there is one, and h's box is refilled when its sums are formed, Pi's after its own.
// Same operations in the same order as the one-point kernel: the same bits. The waits are bounded as in
// rhs_pi_tma_kernel.
#pragma once
#include "rhs_pi_tma.cuh"

namespace tgh {

// The geometry of a launch's tiles. Two shapes: 0 for blocks computed to N + 1 points along some axis, 1 for those of
// N points an axis (PiTile::shape).
struct PiTileShape {
  int TY, TZ;            // rows and planes
  int h_bytes, p_bytes;  // of the boxes
};
struct PiTileGeo {
  PiTileShape shape[2];
  int threads, stages;            // threads 0: the kernel does not apply
  int XB, XC;                     // row pitch, column of i = 0
  int p_off, stage, d_off, smem;  // byte offsets of Pi's box in a stage, of a stage, of the inner sums; all of it
  int tiles_y, tiles_z;           // tiles of a block in shape 0
};

constexpr int PI_TILE_THREADS = 384;      // 12 warps leave 168 registers a thread, enough for a pair's coefficients
constexpr int PI_TILE_SMEM = 227 * 1024;  // one CTA an SM

#define TGH_DECLARE_PI_TILE(QQ)                                                                                   \
  cudaError_t launch_pi_tile_q##QQ(bool diss, int mode, unsigned grid, cudaStream_t s, const RhsArgs& a, const TmaMaps& M, \
                                   WaitStatus st, const PiTileGeo& g, const PiLaunch& L, int tiles);
TGH_DECLARE_PI_TILE(2)
TGH_DECLARE_PI_TILE(4)
TGH_DECLARE_PI_TILE(6)
TGH_DECLARE_PI_TILE(8)

namespace pitile {
template <int Q> struct Rad {
  static constexpr int R = W<Q>::R, KR = W<Q>::RD;
  static constexpr int RP = (R + 1) / 2 * 2, KP = (KR + 1) / 2 * 2;  // in whole pairs
};
// out[i] = column i0 - HP + i of the row at p
template <int HP> __device__ __forceinline__ void load_row(const double* p, double out[2 * HP + 2]) {
#pragma unroll
  for (int t = 0; t <= HP; ++t) {
    const double2 q = lds2(p - HP + 2 * t);
    out[2 * t] = q.x;
    out[2 * t + 1] = q.y;
  }
}
// term-by-term sum over offsets -R..R without the centre, of first-derivative weights (the reference's order)
template <int Q> __device__ __forceinline__ void fold(double2& s, int n, double2 r) {
  constexpr int R = W<Q>::R;
  const int e = n < R ? n - R : n - R + 1;
  const double t0 = __dmul_rn(d1s<Q>(e), r.x), t1 = __dmul_rn(d1s<Q>(e), r.y);
  s.x = n == 0 ? t0 : __dadd_rn(s.x, t0);
  s.y = n == 0 ? t1 : __dadd_rn(s.y, t1);
}
template <int Q> __device__ __forceinline__ double2 inner(const double* p, int s, double2 r[2 * W<Q>::R]) {
  constexpr int R = W<Q>::R;
  double2 in = make_double2(0.0, 0.0);
#pragma unroll
  for (int n = 0; n < 2 * R; ++n) {
    r[n] = lds2(p + (n < R ? n - R : n - R + 1) * s);
    fold<Q>(in, n, r[n]);
  }
  return in;
}
template <int Q> __device__ __forceinline__ void d1_d2(const double2 r[2 * W<Q>::R], double2 c, double d1[2], double d2[2]) {
  constexpr int R = W<Q>::R;
  d1[0] = d1[1] = 0.0;
#pragma unroll
  for (int k = 1; k <= R; ++k) {
    d1[0] = fma(W<Q>::d1(k), r[R - 1 + k].x - r[R - k].x, d1[0]);
    d1[1] = fma(W<Q>::d1(k), r[R - 1 + k].y - r[R - k].y, d1[1]);
  }
  d2[0] = __dmul_rn(W<Q>::d2(R), r[0].x);
  d2[1] = __dmul_rn(W<Q>::d2(R), r[0].y);
#pragma unroll
  for (int k = -R + 1; k <= R; ++k) {
    const double2 u = k == 0 ? c : r[k < 0 ? k + R : k + R - 1];
    const double w = W<Q>::d2(k < 0 ? -k : k);
    d2[0] = __dadd_rn(d2[0], __dmul_rn(w, u.x));
    d2[1] = __dadd_rn(d2[1], __dmul_rn(w, u.y));
  }
}
template <int Q> __device__ __forceinline__ void outer_x(const double* p, double out[2]) {
  constexpr int R = W<Q>::R, RP = Rad<Q>::RP;
  double r[2 * RP + 2];
  load_row<RP>(p, r);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    double o = __dmul_rn(d1s<Q>(-R), r[RP + e - R]);
#pragma unroll
    for (int a = -R + 1; a <= R; ++a) {
      if (a == 0) continue;
      o = __dadd_rn(o, __dmul_rn(d1s<Q>(a), r[RP + e + a]));
    }
    out[e] = o;
  }
}
}  // namespace pitile

template <int Q, bool DISS, int MODE>
__global__ void __launch_bounds__(PI_TILE_THREADS)
    rhs_pi_tile_kernel(const RhsArgs A, const __grid_constant__ TmaMaps M, const WaitStatus stat, const PiTileGeo g, int b0,
                       int ntiles) {
  using namespace pitile;
  constexpr int R = Rad<Q>::R, KR = Rad<Q>::KR, RP = Rad<Q>::RP, KP = Rad<Q>::KP, G = KR;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const unsigned raw = smem_u32(smem_raw);
  const unsigned base = (raw + 127u) & ~127u;
  unsigned char* smem = smem_raw + (base - raw);
  const unsigned bar = base + g.d_off - 64;  // h's mbarriers of the two stages, then Pi's (8 bytes each)
  const int tid = threadIdx.x, XB = g.XB, N1 = A.N1;
  const int tpb = g.tiles_y * g.tiles_z;
  double* const Dy = reinterpret_cast<double*>(smem + g.d_off);
  auto tile_at = [&](int t) {
    if (MODE == MODE_STAGE) return A.ptiles[t];
    const int r = t % tpb;
    return PiTile{b0 + t / tpb, (unsigned char)(r % g.tiles_y * g.shape[0].TY),
                  (unsigned char)(r / g.tiles_y * g.shape[0].TZ), 0, 7};
  };
  // copy n: component n % 10 of the CTA's tile n / 10; its boxes of h and Pi in stage n % stages
  auto stage_of = [&](int n) { return g.stages == 2 ? n & 1 : 0; };
  auto phase_of = [&](int n) { return (unsigned)(g.stages == 2 ? n >> 1 : n) & 1u; };
  auto issue = [&](int n, bool h, bool pi) {
    const int t = blockIdx.x + (n / NC) * gridDim.x;
    if (t >= ntiles) return;
    const PiTile T = tile_at(t);
    const int v = n % NC, st = stage_of(n);
    const unsigned s = base + st * g.stage;
    const PiTileShape sh = g.shape[T.shape];
    const PiMaps& m = T.shape ? M.inner : M.whole;
    if (h) {
      mbar_expect_tx(bar + 8 * st, sh.h_bytes);
      tma_load_4d(s, &m.h, 0, T.y0 + G - R, T.z0 + G - R, T.b * NV + v, bar + 8 * st);
    }
    if (pi) {
      mbar_expect_tx(bar + 16 + 8 * st, sh.p_bytes);
      tma_load_4d(s + g.p_off, &m.pi, 0, T.y0 + G - KR, T.z0 + G - KR, T.b * NV + NC + v, bar + 16 + 8 * st);
    }
  };
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) mbar_init(bar + 8 * i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    issue(0, true, true);
    if (g.stages == 2) issue(1, true, true);
  }
  __syncthreads();

  const long S = (long)N1 * N1 * N1, SX = (long)A.NX * N1 * N1, sv = (long)A.Wx * A.Wd * A.Wd;
  int n = 0, pend_h = g.stages, pend_p = g.stages;  // copies consumed; issued of h and of Pi (thread 0's view)
  bool ok = true;
#pragma unroll 1
  for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x) {
    const PiTile T = tile_at(t);
    const int ex = N1 - 1 + (T.full & 1), ey = N1 - 1 + ((T.full >> 1) & 1), ez = N1 - 1 + (T.full >> 2);
    const int TY = g.shape[T.shape].TY, TZ = g.shape[T.shape].TZ, ROWS = TY * TZ;
    const int HY = TY + 2 * R, PY = TY + 2 * KR, s3h = XB * HY, s3p = XB * PY;
    double* const Dz = Dy + XB * ROWS;
    const int NP = (ex + 1) / 2;
    const bool active = tid < NP * ROWS;
    const int row = active ? tid / NP : 0, i0 = active ? 2 * (tid - row * NP) : 0;
    const int kk = row / TY, jj = row - kk * TY;
    const int c0 = i0 + g.XC;
    const int cH = c0 + XB * ((jj + R) + HY * (kk + R)), cP = c0 + XB * ((jj + KR) + PY * (kk + KR));
    const int cDy = c0 + XB * row, cDz = c0 + XB * ((jj + R) + HY * kk);
    // inner sums beyond the tile's pairs: D_y and D_z RP / 2 pairs beyond each end of its rows, D_z on the R rows
    // either side of it
    const int nx = ROWS * RP, NE = 2 * nx + 2 * R * TZ * NP;
    const int j = T.y0 + jj, k = T.z0 + kk, b = T.b;
    const bool own0 = active && i0 < ex && j < ey && k < ez, own1 = own0 && i0 + 1 < ex;
    const int jc = j < N1 ? j : N1 - 1, kc = k < N1 ? k : N1 - 1;
    const long ic = i0 + (long)A.NX * (jc + (long)N1 * kc);
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
    const long wo = (long)b * NV * sv + (i0 + G) + (long)A.Wx * ((jc + G) + (long)A.Wd * (kc + G));
    double* acc = MODE == MODE_STAGE ? A.acc + (long)b * NV * SX + ic : nullptr;
    double* du = MODE == MODE_DU ? A.du + (long)b * NV * S + i0 + N1 * (jc + (long)N1 * kc) : nullptr;

#pragma unroll 1
    for (int v = 0; v < NC; ++v, ++n) {
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
      const int st = stage_of(n);
      const unsigned ph = phase_of(n);
      // every thread waits (bounded) for h's box; the CTA goes on only if all of them saw it. The vote is also the
      // barrier after the component before: its stage and the inner sums may now be refilled.
      bool got = mbar_wait(bar + 8 * st, ph, stat.first_limit());
      if (!__syncthreads_and(got)) {
        ok = false;
        break;
      }
      if (g.stages == 2 && n >= 1) {
        if (tid == 0) issue(n + 1, true, true);
        pend_h = pend_p = n + 2;
      }
      const double* H = reinterpret_cast<const double*>(smem + st * g.stage);
      const double* P = reinterpret_cast<const double*>(smem + st * g.stage + g.p_off);
      double s[2], p2[2], hd1[3][2], ko[2];
      if (active) {
        const double* hc = H + cH;
        double hx[2 * RP + 2], d2[2];
        load_row<RP>(hc, hx);
        const double2 c = make_double2(hx[RP], hx[RP + 1]);
        double2 r[2 * R];
        *reinterpret_cast<double2*>(Dy + cDy) = inner<Q>(hc, XB, r);
        d1_d2<Q>(r, c, hd1[1], d2);
        p2[0] = d2[0];
        p2[1] = d2[1];
        *reinterpret_cast<double2*>(Dz + cDz) = inner<Q>(hc, s3h, r);
        d1_d2<Q>(r, c, hd1[2], d2);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double* u = hx + RP + e;
          double a = 0.0;
#pragma unroll
          for (int kx = 1; kx <= R; ++kx) a = fma(W<Q>::d1(kx), u[kx] - u[-kx], a);
          hd1[0][e] = a;
          double d = __dmul_rn(W<Q>::d2(R), u[-R]);
#pragma unroll
          for (int kx = -R + 1; kx <= R; ++kx) d = __dadd_rn(d, __dmul_rn(W<Q>::d2(kx < 0 ? -kx : kx), u[kx]));
          double q = cb[e][CF_AXX] * d;
          q = fma(cb[e][CF_AYY], p2[e], q);
          p2[e] = fma(cb[e][CF_AZZ], d2[e], q);
        }
      }
      for (int x = tid; x < NE; x += blockDim.x) {
        int cS, sS;
        double* dst;
        if (x < 2 * nx) {
          // RP pairs a row: RP / 2 left of it, RP / 2 right
          const bool isy = x < nx;
          const int y = isy ? x : x - nx, rr = y / RP, m2 = y - rr * RP;
          const int col = g.XC + (m2 < RP / 2 ? 2 * m2 - RP : 2 * NP + 2 * (m2 - RP / 2));
          const int kz = rr / TY, jy = rr - kz * TY;
          cS = col + XB * ((jy + R) + HY * (kz + R));
          sS = isy ? XB : s3h;
          dst = isy ? Dy + col + XB * rr : Dz + col + XB * ((jy + R) + HY * kz);
        } else {
          const int y = x - 2 * nx, mm = y / NP, col = g.XC + 2 * (y - mm * NP);
          const int kz = mm / (2 * R), jr = mm - kz * (2 * R), jy = jr < R ? jr : jr + TY;
          cS = col + XB * (jy + HY * (kz + R));
          sS = s3h;
          dst = Dz + col + XB * (jy + HY * kz);
        }
        double2 r[2 * R];
        *reinterpret_cast<double2*>(dst) = inner<Q>(H + cS, sS, r);
      }
      if (g.stages == 1) {
        __syncthreads();  // h's box is read
        if (tid == 0) issue(n + 1, true, false);
        pend_h = n + 2;
      }
      got = mbar_wait(bar + 16 + 8 * st, ph, stat.limit);
      if (active && got) {
        const double* pc = P + cP;
        double px[2 * KP + 2], d1[3][2], kd[3][2];
        load_row<KP>(pc, px);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double* u = px + KP + e;
          double a = 0.0;
#pragma unroll
          for (int kx = 1; kx <= R; ++kx) a = fma(W<Q>::d1(kx), u[kx] - u[-kx], a);
          d1[0][e] = a;
          double c = W<Q>::ko(0) * u[0];
          kd[1][e] = kd[2][e] = c;
          if (DISS) {
#pragma unroll
            for (int kx = 1; kx <= KR; ++kx) c = fma(W<Q>::ko(kx), u[kx] + u[-kx], c);
          }
          kd[0][e] = c;
        }
#pragma unroll
        for (int axis = 1; axis < 3; ++axis) {
          const int sx = axis == 1 ? XB : s3p;
          d1[axis][0] = d1[axis][1] = 0.0;
#pragma unroll
          for (int kt = 1; kt <= KR; ++kt) {
            if (!DISS && kt > R) break;
            const double2 u2 = lds2(pc + kt * sx), l2 = lds2(pc - kt * sx);
            if (kt <= R) {
              d1[axis][0] = fma(W<Q>::d1(kt), u2.x - l2.x, d1[axis][0]);
              d1[axis][1] = fma(W<Q>::d1(kt), u2.y - l2.y, d1[axis][1]);
            }
            if (DISS) {
              kd[axis][0] = fma(W<Q>::ko(kt), u2.x + l2.x, kd[axis][0]);
              kd[axis][1] = fma(W<Q>::ko(kt), u2.y + l2.y, kd[axis][1]);
            }
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double* c = cb[e];
          double a = c[CF_B0] * (ih * d1[0][e]);
          a = fma(c[CF_B1], ih * d1[1][e], a);
          a = fma(c[CF_B2], ih * d1[2][e], a);
          a = fma(c[CF_DIVB], px[KP + e], a);
          a = fma(c[CF_DA0], ih * hd1[0][e], a);
          a = fma(c[CF_DA1], ih * hd1[1][e], a);
          s[e] = fma(c[CF_DA2], ih * hd1[2][e], a);
          ko[e] = kd[0][e] + kd[1][e] + kd[2][e];
        }
      }
      // the inner sums are written (and Pi's box is read)
      if (!__syncthreads_and(got)) {
        ok = false;
        break;
      }
      if (g.stages == 1) {
        if (tid == 0) issue(n + 1, false, true);
        pend_p = n + 2;
      }
      if (!any) continue;
      {
        double mxy[2], mxz[2];
        double2 myz = make_double2(0.0, 0.0);
        outer_x<Q>(Dy + cDy, mxy);
        outer_x<Q>(Dz + cDz, mxz);
#pragma unroll
        for (int a = 0; a < 2 * R; ++a) fold<Q>(myz, a, lds2(Dz + cDz + (a < R ? a - R : a - R + 1) * XB));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double* c = cb[e];
          double q = fma(c[CF_AXY], mxy[e], p2[e]);
          q = fma(c[CF_AXZ], mxz[e], q);
          q = fma(c[CF_AYZ], e == 0 ? myz.x : myz.y, q);
          s[e] = fma(ih2, q, s[e]);
          if (DISS) s[e] = fma(c[CF_EH], ko[e], s[e]);
        }
      }
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
  }
  if (!ok) {
    // a wait gave up: record it, let the copies already issued land, bounded, then leave without writing further. With
    // one stage, copy n + 1 of h is issued on the barrier of copy n once that is consumed, and when it has landed a wait
    // for copy n's phase would wait for a copy that is never issued: only copy n + 1 is waited for then.
    if (tid == 0) {
      stat.gave_up();
      auto issued = [&](int c) { return blockIdx.x + (long)(c / NC) * gridDim.x < ntiles; };
      for (int c = g.stages == 1 ? pend_h - 1 : n; c < pend_h; ++c)
        if (issued(c)) mbar_wait(bar + 8 * stage_of(c), phase_of(c), 1ll << 24);
      for (int c = n; c < pend_p; ++c)
        if (issued(c)) mbar_wait(bar + 16 + 8 * stage_of(c), phase_of(c), 1ll << 24);
    }
    __syncthreads();  // the shared arrays outlive their copies
  }
}

template <int Q, bool DISS, int MODE>
cudaError_t launch_pi_tile_t(unsigned grid, cudaStream_t s, const RhsArgs& a, const TmaMaps& M, WaitStatus st,
                             const PiTileGeo& g, const PiLaunch& L, int tiles) {
  if (L.first) {
    const cudaError_t e = cudaFuncSetAttribute(rhs_pi_tile_kernel<Q, DISS, MODE>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, PI_TILE_SMEM);
    if (e != cudaSuccess) return e;
  }
  rhs_pi_tile_kernel<Q, DISS, MODE><<<grid, g.threads, g.smem, s>>>(a, M, st, g, L.b0, tiles);
  return cudaGetLastError();
}
#define TGH_DEFINE_PI_TILE(QQ)                                                                                    \
  cudaError_t launch_pi_tile_q##QQ(bool diss, int mode, unsigned grid, cudaStream_t s, const RhsArgs& a, const TmaMaps& M, \
                                   WaitStatus st, const PiTileGeo& g, const PiLaunch& L, int tiles) {             \
    if (diss) return mode == MODE_DU ? launch_pi_tile_t<QQ, true, MODE_DU>(grid, s, a, M, st, g, L, tiles)                      \
                                     : launch_pi_tile_t<QQ, true, MODE_STAGE>(grid, s, a, M, st, g, L, tiles) ;                 \
    return mode == MODE_DU ? launch_pi_tile_t<QQ, false, MODE_DU>(grid, s, a, M, st, g, L, tiles)                               \
                           : launch_pi_tile_t<QQ, false, MODE_STAGE>(grid, s, a, M, st, g, L, tiles) ;                          \
  }

}  // namespace tgh
