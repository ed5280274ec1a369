// resident_a.cu -- instantiations of the cluster-resident sweeps (resident.cuh) for
// 2 and 4 cells per lane.
#include "resident.cuh"

namespace tomo {
namespace {
template <typename Args>
cudaError_t pick(const ResShape& s, const DevGeo* g, const Args* a, int* held, void* stream) {
    if (s.cpl == 2 && s.rpw == 1) return res_go<2, 1>(s, g, a, held, stream);
    if (s.cpl == 2 && s.rpw == 2) return res_go<2, 2>(s, g, a, held, stream);
    if (s.cpl == 2 && s.rpw == 4) return res_go<2, 4>(s, g, a, held, stream);
    if (s.cpl == 4 && s.rpw == 1) return res_go<4, 1>(s, g, a, held, stream);
    if (s.cpl == 4 && s.rpw == 2) return res_go<4, 2>(s, g, a, held, stream);
    if (s.cpl == 4 && s.rpw == 4) return res_go<4, 4>(s, g, a, held, stream);
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t res_fwd_a(const ResShape& s, const DevGeo* g, const ResFwd* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}
cudaError_t res_adj_a(const ResShape& s, const DevGeo* g, const ResAdj* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}

}  // namespace tomo
