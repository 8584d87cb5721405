// Quadratic mixed mode with a lane per T10 (xfem_qmixed.cuh).
#include "xfem_t10_lane.cuh"
#include "xfem_qmixed.cuh"

namespace xfem {

int launch_qmixed_lane(const DevCtx& ch27, const DevCtx& ct10, uint32_t nsub, float dt, void* stream) {
	return launch_qmixed_of<t10e::T10Lane>(ch27, ct10, nsub, dt, stream);
}

}  // namespace xfem
