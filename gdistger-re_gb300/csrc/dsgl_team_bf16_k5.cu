// The team engine (dsgl_team.cuh) for bf16 tables and up to 5 negatives.
#include "dsgl_team.cuh"

namespace sgns {

template cudaError_t team_d<STORE_BF16, 7>(int d, const TeamCall& c);

}  // namespace sgns
