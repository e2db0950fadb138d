// dsgl_team.cu -- dispatch of the team engine (dsgl_team.cuh): storage x output capacity.
#include "dsgl_team.cuh"

namespace sgns {

extern template cudaError_t team_d<STORE_F32, 7>(int, const TeamCall&);
extern template cudaError_t team_d<STORE_F32, kOMax>(int, const TeamCall&);
extern template cudaError_t team_d<STORE_BF16, 7>(int, const TeamCall&);
extern template cudaError_t team_d<STORE_BF16, kOMax>(int, const TeamCall&);

size_t team_smem_bytes(int d, int window, int K, int lmax, int workers_per_cta) {
  const TeamLayout L = team_layout(d, window, K <= 5 ? 7 : kOMax, lmax);
  return sizeof(float) * ((size_t)kHdrWords + (size_t)workers_per_cta * L.words);
}

namespace {

cudaError_t team_call(int storage, int d, int K, const TeamCall& c) {
  if (storage == STORE_BF16) return K <= 5 ? team_d<STORE_BF16, 7>(d, c) : team_d<STORE_BF16, kOMax>(d, c);
  return K <= 5 ? team_d<STORE_F32, 7>(d, c) : team_d<STORE_F32, kOMax>(d, c);
}

}  // namespace

cudaError_t team_engine_occupancy(int storage, int d, int w, int K, int lmax, int wpc, int* ctas) {
  const TeamCall c{nullptr, wpc, team_smem_bytes(d, w, K, lmax, wpc), ctas, nullptr};
  return team_call(storage, d, K, c);
}

cudaError_t launch_team_engine(const TrainParams& p, int wpc, cudaStream_t s) {
  const TeamCall c{&p, wpc, team_smem_bytes(p.d, p.window, p.K, p.lmax, wpc), nullptr, s};
  return team_call(p.storage, p.d, p.K, c);
}

}  // namespace sgns
