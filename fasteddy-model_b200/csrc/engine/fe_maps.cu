// fe_maps.cu -- tensor maps of the i-marching stage kernel (fe_march_launch.cuh).
#include "fasteddy_b200.h"
#include "fe_march_launch.cuh"

namespace fe {

namespace {
using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                            const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver's encoder through the runtime (no link-time driver dependency).
Encode encoder() {
  static Encode fn = []() -> Encode {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult st;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &st) != cudaSuccess ||
        st != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      return nullptr;
    }
    return (Encode)p;
  }();
  return fn;
}

// Map of nf fields (nf = 0: one field, three dimensions) at field pointer `f` with boxes of bk levels
// by bj rows of one plane and bf fields. The map starts at the row padding, so level k is x = k + ROW_PAD.
bool encode(const Phys& P, const float* f, int nf, int bk, int bj, int bf, CUtensorMap* m) {
  Encode fn = encoder();
  if (!fn) return false;
  const cuuint64_t dim[4] = {(cuuint64_t)P.sj, (cuuint64_t)P.nyh, (cuuint64_t)P.nxh, (cuuint64_t)(nf ? nf : 1)};
  const cuuint64_t stride[3] = {(cuuint64_t)P.sj * 4, (cuuint64_t)P.si * 4, (cuuint64_t)P.n * 4};
  const cuuint32_t box[4] = {(cuuint32_t)bk, (cuuint32_t)bj, 1, (cuuint32_t)bf};
  const cuuint32_t one[4] = {1, 1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, nf ? 4 : 3, const_cast<float*>(f - ROW_PAD), dim, stride, box, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

// (the grid fields and the base state are one allocation each, in these orders: fe_create)
cudaError_t march_encode_maps(const Phys& P, const Ptrs& Q, int tj, const float* cur, const float* pcur,
                              const float* base, MarchMaps* out) {
  const float* sgsF = Q.sgsF;
  const int sgsFields = P.nmoist > 0 ? 7 : 5;
  const bool ok = encode(P, cur, P.nf, 40, tj + 6, 2, &out->ring) && encode(P, cur, P.nf, 32, tj, 2, &out->own) &&
                  encode(P, cur, P.nf, 32, tj, P.nf, &out->ownAll) && encode(P, pcur, 0, 40, tj + 2, 1, &out->pres) &&
                  encode(P, base, P.nf, 32, tj, P.nf, &out->base) &&
                  encode(P, sgsF ? sgsF : cur, sgsF ? sgsFields : P.nf, 32, tj, sgsF ? sgsFields : P.nf, &out->sgs) &&
                  encode(P, Q.zPos, 6, 32, tj, 6, &out->grid) && encode(P, Q.rhoBS, 3, 32, tj, 1, &out->bs);
  return ok ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace fe
