// Host side of the TMA-staged Pi kernel: the tensor maps of a working array and the launch.
#include <cudaTypedefs.h>

#include <string>

#include <algorithm>
#include <cmath>

#include "rhs_pi_tile.cuh"

namespace tgh {

// The working array of nwb blocks (from the start of its allocation: row_lead doubles before its first
// point) viewed as a 4-d tensor (x: the pitch Wx, y and z: Wd, block x 20 + variable), copied in boxes of whole
// rows, y rows and z planes. Rows are a multiple of 32 bytes apart (the copies need 16); rows and planes past a
// block's last read zeros.
static bool make_map(double* work, int nwb, int Wd, int Wx, int y, int z, CUtensorMap* out, std::string& err) {
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      err = "the driver offers no cuTensorMapEncodeTiled";
      return false;
    }
    encode = (PFN_cuTensorMapEncodeTiled_v12000)fn;
  }
  const cuuint64_t dims[4] = {(cuuint64_t)Wx, (cuuint64_t)Wd, (cuuint64_t)Wd, (cuuint64_t)NV * nwb};
  const cuuint64_t strides[3] = {(cuuint64_t)Wx * 8, (cuuint64_t)Wx * Wd * 8, (cuuint64_t)Wx * Wd * Wd * 8};
  const cuuint32_t ones[4] = {1, 1, 1, 1}, box[4] = {(cuuint32_t)Wx, (cuuint32_t)y, (cuuint32_t)z, 1};
  const CUresult r = encode(out, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, work, dims, strides, box, ones,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS) return true;
  err = "cuTensorMapEncodeTiled refused the working array's map (error " + std::to_string((int)r) + ")";
  return false;
}

// the maps of rhs_pi_tma_kernel (q = 4, N = 32)
bool make_tma_maps(double* work, int nwb, TmaMaps* out, std::string& err) {
  using namespace pitma;
  const int Wd = N1 + 2 * G;
  return make_map(work, nwb, Wd, XB, Whole::HY, Whole::HZ, &out->whole.h, err) &&
         make_map(work, nwb, Wd, XB, Whole::PY, Whole::PZ, &out->whole.pi, err) &&
         make_map(work, nwb, Wd, XB, Inner::HY, Inner::HZ, &out->inner.h, err) &&
         make_map(work, nwb, Wd, XB, Inner::PY, Inner::PZ, &out->inner.pi, err);
}

// the maps of rhs_pi_tile_kernel: shape 0 in `whole`, shape 1 in `inner`
bool make_tile_maps(double* work, int nwb, int q, int N, const PiTileGeo& g, TmaMaps* out, std::string& err) {
  const int R = q / 2, KR = R + 1, Wd = N + 1 + 2 * KR;
  for (int i = 0; i < 2; ++i) {
    PiMaps& m = i ? out->inner : out->whole;
    const PiTileShape& s = g.shape[i];
    if (!make_map(work, nwb, Wd, g.XB, s.TY + 2 * R, s.TZ + 2 * R, &m.h, err) ||
        !make_map(work, nwb, Wd, g.XB, s.TY + 2 * KR, s.TZ + 2 * KR, &m.pi, err))
      return false;
  }
  return true;
}

// The tile geometry of rhs_pi_tile_kernel for nwhole blocks computed to N + 1 points along some axis and ninner of N
// points an axis, at order q on `sms` SMs; false where none fits (the one-point kernel then runs). Over the tiles of
// at most the kernel's threads in pairs whose boxes and inner sums fit the shared memory it takes, for each shape, the
// least modelled time: the waves of tiles, each taking a component a fixed latency (its waits and barriers, as long
// as 250 pairs' arithmetic) and a time by its pairs and by the doubles it stages (0.02 of a pair each).
// One CTA an SM: two of at most 256 threads, at 128 registers with spills, were slower at every size but the
// smallest (64 blocks of 24^3 at q = 4: 662 us a right-hand side against 536; 27 of 27^3 at q = 8: 530 against 471).
bool pi_tile_geometry(int q, int N, int nwhole, int ninner, int sms, PiTileGeo* out) {
  if (N > 96) return false;
  const int R = q / 2, KR = R + 1, N1 = N + 1, XB = row_pitch(N1 + 2 * KR, KR);
  auto up = [](int b) { return (b + 127) / 128 * 128; };
  double best = 0.0;
  bool found = false;
  for (const int stages : {2, 1}) {
    PiTileGeo g{};
    g.stages = stages;
    g.XB = XB;
    g.XC = row_lead(KR) + KR;
    double total = 0.0;
    const double nb1 = nwhole + ninner;
    int hmax = 0, pmax = 0, dmax = 0;
    bool ok = true;
    for (int i = 0; i < 2 && ok; ++i) {
      const int e = i ? N : N1, NP = (e + 1) / 2, nb = i ? ninner : nwhole + ninner;  // the plain form: all in shape 0
      double least = 0.0;
      PiTileShape sel{};
      int seld = 0;
      for (int ty = 1; ty <= e && NP * ty <= PI_TILE_THREADS; ++ty)
        for (int tz = 1; tz <= e && NP * ty * tz <= PI_TILE_THREADS; ++tz) {
          const int h = 8 * XB * (ty + 2 * R) * (tz + 2 * R), p = 8 * XB * (ty + 2 * KR) * (tz + 2 * KR);
          const int d = 8 * XB * (ty * tz + (ty + 2 * R) * tz);
          if (stages * (up(std::max(h, hmax)) + up(std::max(p, pmax))) + 128 + std::max(d, dmax) + 128 > PI_TILE_SMEM) continue;
          const double waves = std::max(1.0, std::ceil((double)nb * ((e + ty - 1) / ty) * ((e + tz - 1) / tz) / sms));
          const double cost =
              waves * (250.0 + NP * ty * tz + 0.02 * (h + p) / 8) * (stages == 1 ? 1.15 : 1.0);
          if (sel.TY == 0 || cost < least) {
            least = cost;
            sel = PiTileShape{ty, tz, h, p};
            seld = d;
          }
        }
      if (sel.TY == 0) ok = false;
      g.shape[i] = sel;
      g.threads = std::max(g.threads, (NP * sel.TY * sel.TZ + 31) / 32 * 32);
      hmax = std::max(hmax, sel.h_bytes);
      pmax = std::max(pmax, sel.p_bytes);
      dmax = std::max(dmax, seld);
      total += least * (i ? ninner : nwhole) / nb1;
    }
    if (!ok) continue;
    g.p_off = up(hmax);
    g.stage = g.p_off + up(pmax);
    g.d_off = stages * g.stage + 128;  // the mbarriers sit in the 64 bytes before it
    g.smem = g.d_off + dmax + 128;
    g.tiles_y = (N1 + g.shape[0].TY - 1) / g.shape[0].TY;
    g.tiles_z = (N1 + g.shape[0].TZ - 1) / g.shape[0].TZ;
    if (!found || total < best) {
      found = true;
      best = total;
      *out = g;
    }
  }
  return found;
}

template <bool DISS, int MODE>
static cudaError_t launch_pi_tma_t(cudaStream_t s, const RhsArgs& a, const TmaMaps& M, WaitStatus st, const PiLaunch& L) {
  using namespace pitma;
  if (L.first) {
    const cudaError_t e = cudaFuncSetAttribute(rhs_pi_tma_kernel<DISS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               SMEM);
    if (e != cudaSuccess) return e;
  }
  const int tiles = MODE == MODE_STAGE ? a.nptiles : L.nb * TILES;
  rhs_pi_tma_kernel<DISS, MODE><<<(unsigned)std::min(tiles, L.sms), THREADS, SMEM, s>>>(a, M, st, L.b0, tiles);
  return cudaGetLastError();
}

// The Pi kernel over the whole blocks of the launch (q = 4, N = 32, FP64).
cudaError_t launch_pi_tma(bool diss, int mode, cudaStream_t s, const RhsArgs& a, const TmaMaps& M, WaitStatus st,
                          const PiLaunch& L) {
  if (diss) return mode == MODE_DU ? launch_pi_tma_t<true, MODE_DU>(s, a, M, st, L)
                                   : launch_pi_tma_t<true, MODE_STAGE>(s, a, M, st, L);
  return mode == MODE_DU ? launch_pi_tma_t<false, MODE_DU>(s, a, M, st, L)
                         : launch_pi_tma_t<false, MODE_STAGE>(s, a, M, st, L);
}

// The tile Pi kernel over the whole blocks of the launch (FP64).
cudaError_t launch_pi_tile(int q, bool diss, int mode, cudaStream_t s, const RhsArgs& a, const TmaMaps& M, WaitStatus st,
                           const PiTileGeo& g, const PiLaunch& L) {
  const int tiles = mode == MODE_STAGE ? a.nptiles : L.nb * g.tiles_y * g.tiles_z;
  const unsigned grid = (unsigned)std::min(tiles, L.sms);
  switch (q) {
    case 2: return launch_pi_tile_q2(diss, mode, grid, s, a, M, st, g, L, tiles);
    case 4: return launch_pi_tile_q4(diss, mode, grid, s, a, M, st, g, L, tiles);
    case 6: return launch_pi_tile_q6(diss, mode, grid, s, a, M, st, g, L, tiles);
    default: return launch_pi_tile_q8(diss, mode, grid, s, a, M, st, g, L, tiles);
  }
}

}  // namespace tgh
