// resident_e.cu -- instantiations of the cluster-resident reference-profile sweeps
// (resident_ref.cuh) for 4 and 6 cells per lane.
#include "resident_ref.cuh"

namespace tomo {
namespace {
template <typename Args>
cudaError_t pick(const ResShape& s, const DevGeo* g, const Args* a, int* held, void* stream) {
    if (s.cpl == 4) return ref_go<4>(s, g, a, held, stream);
    if (s.cpl == 6) return ref_go<6>(s, g, a, held, stream);
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t res_fwd_e(const ResShape& s, const DevGeo* g, const ResFwd* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}
cudaError_t res_adj_e(const ResShape& s, const DevGeo* g, const ResAdj* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}

}  // namespace tomo
