// The quadratic-tet mode's element kernel with a lane per T10 (launch_t10,
// xfem_t10.cu).
#include "xfem_t10_lane.cuh"

namespace xfem {

int launch_t10_lane(const DevCtx& ctx, uint32_t nsub, float dt, void* stream) {
	return launch_elements<t10e::T10Lane>(ctx, nsub, dt, stream);
}

}  // namespace xfem
