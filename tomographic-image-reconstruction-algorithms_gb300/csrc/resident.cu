// resident.cu -- host side of the cluster-resident sweeps (resident.cuh): which problems they take,
// the shapes their clusters can have, and the receiver tables they read.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "internal.h"

namespace tomo {

#define RES_WIDTHS(X) X(a) X(b) X(c) X(d) X(e) X(f)
#define RES_DECL(W)                                                                                        \
    cudaError_t res_fwd_##W(const ResShape& s, const DevGeo* g, const ResFwd* a, int* held, void* stream); \
    cudaError_t res_adj_##W(const ResShape& s, const DevGeo* g, const ResAdj* a, int* held, void* stream);
RES_WIDTHS(RES_DECL)

namespace {
constexpr int kMaxCluster = 16;

// Cells per lane of a grid width (0: too wide).  Shapes are limited by registers: the adjoint keeps
// z, the previous z, its products and the correlation, 4 x cells per thread, beside about 90 others,
// so a block of up to 8 warps (255 registers) takes 32 cells per thread and one of up to 16 warps
// (128 registers) 16.  The builds of up to 16 warps with the most cells spill (-Xptxas -v, bytes stored / loaded:
// reference forward 10 cells per lane 512 / 784, 8 cells 196 / 288, adjoint 172 / 312 and 60 / 64; CFG adjoint 2 rows of
// 8, 4 of 4 and 1 of 16 cells 110 to 130 / 160 to 190).  A context times its shapes, so they run only where they are
// the faster ones; the allocation-free forward takes its shape untimed, and for reference grids of 288 rows has no
// other.  A 512 x 512 grid would need 64 cells per thread on 16 blocks: tried, it
// spills (41 us per adjoint step of 32 groups against 26 us in the strip kernels and 22 streamed), so such
// grids are streamed or stay with the strip and tile kernels.
int cells_per_lane(int nx) {
    for (const int c : {2, 4, 6, 8, 10, 12, 16})
        if (nx <= 32 * c) return c;
    return 0;
}
cudaError_t fwd(const ResShape& s, const DevGeo* g, const ResFwd* a, int* held, void* st) {
    if (s.ref) return s.cpl <= 6 ? res_fwd_e(s, g, a, held, st) : res_fwd_f(s, g, a, held, st);
    return s.cpl <= 4 ? res_fwd_a(s, g, a, held, st) : s.cpl <= 8 ? res_fwd_b(s, g, a, held, st)
         : s.cpl <= 12 ? res_fwd_c(s, g, a, held, st) : res_fwd_d(s, g, a, held, st);
}
cudaError_t adj(const ResShape& s, const DevGeo* g, const ResAdj* a, int* held, void* st) {
    if (s.ref) return s.cpl <= 6 ? res_adj_e(s, g, a, held, st) : res_adj_f(s, g, a, held, st);
    return s.cpl <= 4 ? res_adj_a(s, g, a, held, st) : s.cpl <= 8 ? res_adj_b(s, g, a, held, st)
         : s.cpl <= 12 ? res_adj_c(s, g, a, held, st) : res_adj_d(s, g, a, held, st);
}

// Largest number of receivers in a band of `rows` rows.
int band_receivers(const std::vector<int32_t>& rowstart, int ny, int rows) {
    int most = 0;
    for (int j = 0; j < ny; j += rows) most = std::max(most, rowstart[std::min(ny, j + rows)] - rowstart[j]);
    return most;
}
}  // namespace

int64_t res_slice(const ResShape& s, int ny) { return (int64_t)32 * s.cpl * ny; }

// Reference profile: cells per lane of a width (0: too wide).
static int ref_cells_per_lane(int nx) {
    for (const int c : {4, 6, 8, 10})
        if (nx <= 32 * c) return c;
    return 0;
}

std::vector<int32_t> ref_warps(int ny, int lo, int hi) {
    std::vector<int32_t> out;
    if (lo < 2 || hi < lo + 3 || hi > ny - 3) return out;   // the paired rows must be four distinct pairs
    auto rows = [&](int a, int b) {                          // rows a .. b-1: pairs, an odd one alone
        for (int j = a; j < b; j += 2) out.push_back(j | (std::min(2, b - j) << 16));
    };
    rows(0, 2);
    rows(2, lo);
    rows(lo, lo + 2);
    rows(lo + 2, hi - 1);
    rows(hi - 1, hi + 1);
    rows(hi + 1, ny - 2);
    rows(ny - 2, ny);
    return out;
}

std::vector<ResShape> ref_shapes(int nx, int ny, const std::vector<int32_t>& warps, const std::vector<int32_t>& rowstart) {
    std::vector<ResShape> out;
    const int cpl = ref_cells_per_lane(nx), nw = (int)warps.size();
    if (cpl == 0 || nw == 0 || ny > 0x7fff) return out;
    for (int cs = kMaxCluster; cs >= 1; --cs) {
        ResShape s;
        s.ref = true;
        s.cpl = cpl;
        s.rpw = 2;
        s.cs = cs;
        s.warps = (nw + cs - 1) / cs;
        if (s.warps > 16 || s.warps * (cs - 1) >= nw) continue;
        for (int b = 0; b < cs; ++b) {
            const int first = warps[b * s.warps], last = warps[std::min(nw, (b + 1) * s.warps) - 1];
            s.nrec = std::max(s.nrec, rowstart[(last & 0xffff) + (last >> 16)] - rowstart[first & 0xffff]);
        }
        out.push_back(s);
    }
    return out;
}
int res_restart(int k0, int K, int ch) { return ch * K + 1 - ((ch * K + 1 - k0) & 1); }

std::vector<ResShape> res_shapes(int nx, int ny, const std::vector<int32_t>& rowstart) {
    std::vector<ResShape> out;
    const int cpl = cells_per_lane(nx);
    if (cpl == 0) return out;
    for (const int rpw : {1, 2, 4})
        for (int cs = kMaxCluster; cs >= 1; --cs) {
            const int warps = ((ny + cs - 1) / cs + rpw - 1) / rpw;
            const int most = cpl * rpw <= 16 ? 16 : cpl * rpw <= 32 ? 8 : 0;
            if (warps > most || (int64_t)warps * rpw * (cs - 1) >= ny) continue;
            ResShape s;
            s.cpl = cpl;
            s.rpw = rpw;
            s.warps = warps;
            s.cs = cs;
            s.nrec = band_receivers(rowstart, ny, s.rows());
            out.push_back(s);
        }
    return out;
}

int res_held(const ResShape& s) {
    int f = 0, b = 0;
    if (fwd(s, nullptr, nullptr, &f, nullptr) == cudaSuccess && adj(s, nullptr, nullptr, &b, nullptr) == cudaSuccess)
        return std::min(f, b);
    cudaGetLastError();
    return 0;
}

ResShape res_pick(const std::vector<ResShape>& shapes, int ng) {
    ResShape best;
    const int want = std::max(1, std::min(kMaxCluster, 144 / std::max(1, ng)));
    for (const ResShape& s : shapes) {
        const bool few = s.cs <= want, best_few = best.cpl && best.cs <= want;
        const bool better = few != best_few ? few : few ? s.cs > best.cs : s.cs < best.cs;
        if (best.cpl == 0 || better) best = s;
    }
    return best;
}

void res_receivers(const std::vector<int32_t>& rcv, int nx, int ny, std::vector<int32_t>& chan,
                   std::vector<int32_t>& cell, std::vector<int32_t>& rowstart) {
    chan.clear();
    for (size_t c = 0; c < rcv.size(); ++c)
        if (rcv[c] >= 0) chan.push_back((int32_t)c);
    std::stable_sort(chan.begin(), chan.end(), [&](int32_t a, int32_t b) { return rcv[a] < rcv[b]; });
    cell.clear();
    for (const int32_t c : chan) cell.push_back(rcv[c]);
    rowstart.assign((size_t)ny + 1, 0);
    for (const int32_t q : cell) ++rowstart[(size_t)(q / nx) + 1];
    for (int j = 0; j < ny; ++j) rowstart[j + 1] += rowstart[j];
}

void launch_res_fwd(const ResShape& s, const DevGeo& g, const ResFwd& a, void* stream) { fwd(s, &g, &a, nullptr, stream); }
void launch_res_adj(const ResShape& s, const DevGeo& g, const ResAdj& a, void* stream) { adj(s, &g, &a, nullptr, stream); }

}  // namespace tomo
