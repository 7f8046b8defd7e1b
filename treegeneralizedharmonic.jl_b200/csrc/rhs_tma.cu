// Host side of the TMA-staged Pi kernel: the tensor maps of a working array and the launch.
#include <cudaTypedefs.h>

#include <cstring>
#include <string>

#include "rhs_pi_tma.cuh"

namespace tgh {

// The working array of nwb blocks (from the start of its allocation: row_lead doubles before its first
// point) viewed as a 4-d tensor (x: the pitch Wx = 40, y: 39, z: 39, block x 20 + variable). Rows are
// 320 bytes apart (a multiple of 16, as the copies need), and the boxes are whole rows; rows and
// planes past a block's last read zeros.
bool make_tma_maps(double* work, int nwb, TmaMaps* out, std::string& err) {
  using namespace pitma;
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
  const int Wd = N1 + 2 * G, Wx = row_pitch(Wd, G);
  const cuuint64_t dims[4] = {(cuuint64_t)Wx, (cuuint64_t)Wd, (cuuint64_t)Wd, (cuuint64_t)NV * nwb};
  const cuuint64_t strides[3] = {(cuuint64_t)Wx * 8, (cuuint64_t)Wx * Wd * 8, (cuuint64_t)Wx * Wd * Wd * 8};
  const cuuint32_t ones[4] = {1, 1, 1, 1};
  auto map = [&](CUtensorMap* m, int x, int y, int z) {
    const cuuint32_t box[4] = {(cuuint32_t)x, (cuuint32_t)y, (cuuint32_t)z, 1};
    return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, work, dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  };
  CUresult r = map(&out->whole.h, XB, Whole::HY, Whole::HZ);
  if (r == CUDA_SUCCESS) r = map(&out->whole.pi, XB, Whole::PY, Whole::PZ);
  if (r == CUDA_SUCCESS) r = map(&out->inner.h, XB, Inner::HY, Inner::HZ);
  if (r == CUDA_SUCCESS) r = map(&out->inner.pi, XB, Inner::PY, Inner::PZ);
  if (r != CUDA_SUCCESS) {
    err = "cuTensorMapEncodeTiled refused the working array's map (error " + std::to_string((int)r) + ")";
    return false;
  }
  return true;
}

static cudaError_t sm_count(int* sms) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  return e == cudaSuccess ? cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev) : e;
}

template <bool DISS, int MODE>
static cudaError_t launch_pi_tma_t(cudaStream_t s, const RhsArgs& a, const TmaMaps& M, WaitStatus st, int b0,
                                   int nb) {
  using namespace pitma;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(rhs_pi_tma_kernel<DISS, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         SMEM);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  int sms = 0;
  cudaError_t e = sm_count(&sms);
  if (e != cudaSuccess) return e;
  const int tiles = MODE == MODE_STAGE ? a.nptiles : nb * TILES;
  rhs_pi_tma_kernel<DISS, MODE><<<(unsigned)(tiles < sms ? tiles : sms), THREADS, SMEM, s>>>(a, M, st, b0, tiles);
  return cudaGetLastError();
}

// The Pi kernel over the whole blocks b0 .. b0 + nb - 1 (q = 4, N = 32, FP64).
cudaError_t launch_pi_tma(bool diss, int mode, cudaStream_t s, const RhsArgs& a, const TmaMaps& M, WaitStatus st,
                          int b0, int nb) {
  if (diss) return mode == MODE_DU ? launch_pi_tma_t<true, MODE_DU>(s, a, M, st, b0, nb)
                                   : launch_pi_tma_t<true, MODE_STAGE>(s, a, M, st, b0, nb);
  return mode == MODE_DU ? launch_pi_tma_t<false, MODE_DU>(s, a, M, st, b0, nb)
                         : launch_pi_tma_t<false, MODE_STAGE>(s, a, M, st, b0, nb);
}

}  // namespace tgh
