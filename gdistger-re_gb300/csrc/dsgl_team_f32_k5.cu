// The team engine (dsgl_team.cuh) for fp32 tables and up to 5 negatives.
#include "dsgl_team.cuh"

namespace sgns {

template cudaError_t team_d<STORE_F32, 7>(int d, const TeamCall& c);

}  // namespace sgns
