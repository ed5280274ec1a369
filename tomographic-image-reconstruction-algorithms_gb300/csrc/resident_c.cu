// resident_c.cu -- instantiations of the cluster-resident sweeps (resident.cuh) for
// 10 and 12 cells per lane.
#include "resident.cuh"

namespace tomo {
namespace {
template <typename Args>
cudaError_t pick(const ResShape& s, const DevGeo* g, const Args* a, int* held, void* stream) {
    if (s.cpl == 10 && s.rpw == 1) return res_go<10, 1>(s, g, a, held, stream);
    if (s.cpl == 10 && s.rpw == 2) return res_go<10, 2>(s, g, a, held, stream);
    if (s.cpl == 12 && s.rpw == 1) return res_go<12, 1>(s, g, a, held, stream);
    if (s.cpl == 12 && s.rpw == 2) return res_go<12, 2>(s, g, a, held, stream);
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t res_fwd_c(const ResShape& s, const DevGeo* g, const ResFwd* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}
cudaError_t res_adj_c(const ResShape& s, const DevGeo* g, const ResAdj* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}

}  // namespace tomo
