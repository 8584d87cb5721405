// Quadratic mixed mode with four lanes per T10 (xfem_qmixed.cuh).
#include "xfem_t10_elem.cuh"
#define XFEM_H27_SMEM_AT sizeof(t10e::QuadShared)
#include "xfem_qmixed.cuh"

namespace xfem {

int launch_qmixed(const DevCtx& ch27, const DevCtx& ct10, int t10_lanes, uint32_t nsub, float dt, void* stream) {
	return t10_lanes == 4 ? launch_qmixed_of<t10e::T10Elem>(ch27, ct10, nsub, dt, stream)
	                      : launch_qmixed_lane(ch27, ct10, nsub, dt, stream);
}

}  // namespace xfem
