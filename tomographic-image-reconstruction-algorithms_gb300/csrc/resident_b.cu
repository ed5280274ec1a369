// resident_b.cu -- instantiations of the cluster-resident sweeps (resident.cuh) for
// 6 and 8 cells per lane.
#include "resident.cuh"

namespace tomo {
namespace {
template <typename Args>
cudaError_t pick(const ResShape& s, const DevGeo* g, const Args* a, int* held, void* stream) {
    if (s.cpl == 6 && s.rpw == 1) return res_go<6, 1>(s, g, a, held, stream);
    if (s.cpl == 6 && s.rpw == 2) return res_go<6, 2>(s, g, a, held, stream);
    if (s.cpl == 6 && s.rpw == 4) return res_go<6, 4>(s, g, a, held, stream);
    if (s.cpl == 8 && s.rpw == 1) return res_go<8, 1>(s, g, a, held, stream);
    if (s.cpl == 8 && s.rpw == 2) return res_go<8, 2>(s, g, a, held, stream);
    if (s.cpl == 8 && s.rpw == 4) return res_go<8, 4>(s, g, a, held, stream);
    return cudaErrorInvalidValue;
}
}  // namespace

cudaError_t res_fwd_b(const ResShape& s, const DevGeo* g, const ResFwd* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}
cudaError_t res_adj_b(const ResShape& s, const DevGeo* g, const ResAdj* a, int* held, void* stream) {
    return pick(s, g, a, held, stream);
}

}  // namespace tomo
