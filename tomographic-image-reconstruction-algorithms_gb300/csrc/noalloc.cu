// noalloc.cu -- forward solve into caller-owned device buffers with no device
// allocation at all (tomo_forward_noalloc in include/tomo.h).
//
// Why it exists: tomo_create sizes and cudaMallocs a context.  Some callers
// cannot do that -- a host application that hands every byte of device memory
// to its own pool allocator and forbids raw cudaMalloc, or a latency-bound loop
// where cudaMalloc/cudaFree would synchronise the device and stall its other
// streams.  They pass their own input and output buffers; the wavefield
// scratch this solve needs lives in the file-scope array below instead.
//
// Grids that fit on chip (resident.cuh) are solved by one launch for all groups, which keeps the
// wavefield in registers and uses the array for the coefficients and tables only: 128 x 128, 600
// steps, 8 groups took 39.2 ms as a step and a gather launch per time step and group and takes 0.24.
// Larger grids go a group at a time through the array's time slots: benchmark-profile grids whose framed
// slices fit the array by the streamed sweeps, four steps to a launch (launches are what bounds it; 300 x 330
// 8.2 -> 3.8 us per step and group), the others by a step and a gather launch per time step.
//
// The scratch array g_scratch is a fixed kNoallocScratchBytes (about 5.6 MiB)
// that every GPU loading this library holds until the process exits.  It holds
// the coefficient fields, the geometry tables and, for one emitter group at
// a time, three forward time slots (four framed ones in a streamed solve), so a call accepts grids of up to
// kNoallocMaxCells cells (512 x 512), kNoallocMaxChannels record channels and
// kNoallocMaxSteps time steps, plus kNoallocMaxEmitters emitters (benchmark
// profile) or kNoallocMaxGroups emission boxes (reference profile), and rejects
// anything larger with TOMO_ERR_ARG.
//
// In host code g_scratch names a host-side stand-in, not device memory.  Every
// call looks the array's device address up with cudaGetSymbolAddress on the
// current device and passes that pointer to the kernels, so the address is
// right for whatever context is current (also after a cudaDeviceReset, which
// reloads the module at a new address).  The first call on a device also loads
// the module's code there: make that first call before any stream capture.
//
// The geometry tables travel to the array as kernel arguments (k_put_words),
// not as copies from host memory, so nothing on the device side refers to the
// call's host-side tables after it returns.
//
// All calls share the one array and it keeps the last call's contents: each
// call zeroes the time slots it starts from and the output records,
// and rewrites everything else before reading it.  The blocks of a cluster wait for each other's rows, at most
// a second; the call has returned by then, so a group whose wait runs out leaves NaN in all its records.  Calls that overlap on the
// GPU (concurrent streams, or threads, on the same device) race on the array:
// serialise them on one stream.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include "internal.h"

namespace tomo {
namespace {

constexpr int64_t kNoallocMaxCells = 512 * 512;
constexpr int kNoallocMaxChannels = 2048;
constexpr int kNoallocMaxGroups = 2048;
constexpr int kNoallocMaxEmitters = 4096;
constexpr int kNoallocMaxSteps = 16384;
constexpr int kNoallocMaxRows = 1024;      // grid rows of a cluster-resident solve

// float region: 3 time slots + coefficient + edge coefficient, or the framed slots and coefficient of a streamed
// solve (528 x 536 + 128 floats each at 512 x 512); then the source table
constexpr int64_t kFields = 5 * (int64_t)(528 * 536 + 128);
constexpr int64_t kFloats = kFields + kNoallocMaxSteps;
static_assert(kFields >= 5 * kNoallocMaxCells, "fields of the largest grid");
// int region: receiver cells, emitter cells, emission boxes; for a cluster-resident solve receivers in row
// order (channel, cell), the first of each row, and the reference profile's rows of each warp and row slots
constexpr int64_t kInts = 3 * kNoallocMaxChannels + kNoallocMaxEmitters + 4 * kNoallocMaxGroups + 3 * (kNoallocMaxRows + 1);
constexpr int64_t kNoallocScratchBytes = 4 * (kFloats + kInts);

static __device__ __align__(256) unsigned char g_scratch[kNoallocScratchBytes];

// Words of table data carried by one k_put_words launch (the argument block stays under the 32764-byte
// kernel-parameter limit): most problems' tables go in one launch.
constexpr int kWordsPerLaunch = 4000;
struct Words {
    uint32_t v[kWordsPerLaunch];
};

__global__ void k_put_words(uint32_t* __restrict__ dst, int n, Words w) {
    for (int t = threadIdx.x; t < n; t += blockDim.x) dst[t] = w.v[t];
}

// Failures are returned as a status and explained in one line on stderr.
tomo_status fail(tomo_status s, const std::string& why) {
    std::fprintf(stderr, "tomo_forward_noalloc: %s\n", why.c_str());
    return s;
}

tomo_status cuda_fail(cudaError_t e, const char* what) {
    return fail(TOMO_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

// Device address of g_scratch in the current device's context, looked up on every call.
tomo_status scratch_address(unsigned char** out) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);
    if (e != cudaSuccess || !p) return cuda_fail(e, "cudaGetSymbolAddress(g_scratch)");
    *out = (unsigned char*)p;
    return TOMO_OK;
}

// Writes n 32-bit words from host memory to dst on `st`, kWordsPerLaunch per launch, through
// kernel arguments: the words are captured at launch, so `src` may go out of scope on return.
tomo_status put_words(uint32_t* dst, const void* src, int64_t n, cudaStream_t st) {
    Words w;
    const uint32_t* s = (const uint32_t*)src;
    for (int64_t off = 0; off < n; off += kWordsPerLaunch) {
        const int m = (int)std::min<int64_t>(kWordsPerLaunch, n - off);
        std::memcpy(w.v, s + off, sizeof(uint32_t) * m);
        k_put_words<<<1, 256, 0, st>>>(dst + off, m, w);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return cuda_fail(e, "k_put_words");
    }
    return TOMO_OK;
}

}  // namespace
}  // namespace tomo

using namespace tomo;

// A function-try-block: a C++ exception below it (host allocation failure) becomes a status.
extern "C" tomo_status tomo_forward_noalloc(const tomo_config* cfg, const float* d_f, float* d_records,
                                            void* stream) try {
    if (!cfg || !d_f || !d_records) return fail(TOMO_ERR_ARG, "NULL argument");
    Geometry geo;
    std::string why;
    tomo_status s = build_geometry(*cfg, geo, why);
    if (s != TOMO_OK) return fail(s, why);
    // the emitter table is read by the benchmark profile only, the emission boxes by the reference profile
    if (geo.N > kNoallocMaxCells || geo.nch > kNoallocMaxChannels || geo.nt > kNoallocMaxSteps ||
        (geo.ref && geo.G > kNoallocMaxGroups) || (!geo.ref && (int64_t)geo.G * geo.gs > kNoallocMaxEmitters))
        return fail(TOMO_ERR_ARG, "problem exceeds the allocation-free limits (cells <= 262144, channels <= 2048, "
                                  "steps <= 16384, emitters <= 4096, reference-profile groups <= 2048)");
    unsigned char* base = nullptr;
    if ((s = scratch_address(&base)) != TOMO_OK) return s;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t N = geo.N, nt = geo.nt, nch = geo.nch;
    float* slots = (float*)base;                       // 3 time slots
    float* coef = slots + 3 * kNoallocMaxCells;
    float* rcoef = coef + kNoallocMaxCells;
    float* src = slots + kFields;                      // tables: source, then the integer tables behind it
    cudaError_t e;
#define NA_CU(x)                                     \
    do {                                             \
        if ((e = (x)) != cudaSuccess) return cuda_fail(e, #x); \
    } while (0)
    DevGeo dg{};
    dg.nx = geo.nx; dg.ny = geo.ny; dg.nt = geo.nt; dg.nch = geo.nch;
    dg.lo = geo.lo; dg.hi = geo.hi; dg.gs = geo.gs;
    dg.sponge_w = cfg->sponge_width; dg.sponge_max = cfg->sponge_max;
    fill_damp(dg);
    dg.n_src_steps = geo.n_src_steps;
    dg.src = src;
    const int prof = cfg->profile;
    // a grid that fits on chip is solved by one launch for all groups
    std::vector<int32_t> chan, cell, rowstart, warps, slot;
    ResShape shape;
    bool streamed = false;
    if (const char* off = std::getenv("TOMO_RESIDENT"); geo.ny <= kNoallocMaxRows && !(off && *off == '0')) {
        res_receivers(geo.rcv, geo.nx, geo.ny, chan, cell, rowstart);
        if (geo.ref) warps = ref_warps(geo.ny, geo.lo, geo.hi);
        shape = res_pick(geo.ref ? ref_shapes(geo.nx, geo.ny, warps, rowstart) : res_shapes(geo.nx, geo.ny, rowstart), geo.G);
        if (shape.cpl && res_held(shape) < 1) shape = ResShape{};
        streamed = !shape.cpl && !geo.ref && (STREAM_RING + 1) * stream_slice(geo.nx, geo.ny) <= kFields;
    }
    // every table in one block of words behind the source table
    std::vector<uint32_t> words;
    auto put = [&](const void* p, int64_t n) {         // returns the table's device address
        const uint32_t* w = (const uint32_t*)p;
        const int64_t at = (int64_t)words.size();
        words.insert(words.end(), w, w + n);
        return (int32_t*)src + at;
    };
    put(geo.src.data(), shape.cpl ? std::min<int64_t>((int64_t)geo.src.size(), geo.ref ? 2 * geo.n_src_steps : geo.n_src_steps)
                                  : (int64_t)geo.src.size());
    if (geo.ref) dg.box = put(geo.box.data(), 4 * (int64_t)geo.G);
    else dg.emit = put(geo.emit.data(), (int64_t)geo.G * geo.gs);
    ResFwd r{};
    if (shape.cpl || streamed) {
        r.rchan = put(chan.data(), (int64_t)chan.size());
        r.rcell = put(cell.data(), (int64_t)cell.size());
        r.rowstart = put(rowstart.data(), geo.ny + 1);
        if (geo.ref) {
            slot.assign((size_t)geo.ny, 0);
            for (size_t w = 0; w < warps.size(); ++w)
                for (int k = 0; k < warps[w] >> 16; ++k) slot[(warps[w] & 0xffff) + k] = (int32_t)(2 * w) + k;
            r.warps = put(warps.data(), (int64_t)warps.size());
            r.rowslot = put(slot.data(), geo.ny);
            r.nwarps = (int)warps.size();
        }
    } else {
        dg.rcv = put(geo.rcv.data(), nch);
    }
    // the word the kernels' bounded waits set; the caller learns of them by the records (nan_on_timeout)
    static const uint32_t zero = 0;
    unsigned int* const err = (unsigned int*)put(&zero, 1);
    if ((s = put_words((uint32_t*)src, words.data(), (int64_t)words.size(), st)) != TOMO_OK) return s;
    NA_CU(cudaMemsetAsync(d_records, 0, sizeof(float) * (size_t)geo.G * nt * nch, st));
    if (streamed) {
        const int64_t ns = stream_slice(geo.nx, geo.ny);
        float* const framed = slots + STREAM_RING * ns;
        launch_coef(prof, d_f, slots, slots + N, N, cfg->courant, st);   // in the slots' place
        launch_frame(framed, slots, geo.nx, geo.ny, st);
        launch_zero_slots(slots, 1, STREAM_RING * ns, 0, 2 * ns, 2 * ns, st);   // all four, guard cells included
        StreamFwd a{};
        a.coef = framed;
        a.ns = ns;
        a.k0 = 1;
        a.ng = 1;
        a.px = stream_pitch(geo.nx);
        a.rec = StreamRec{r.rchan, r.rcell, r.rowstart};
        for (int g = 0; g < geo.G; ++g) {
            if (g > 0) launch_zero_slots(slots, 1, STREAM_RING * ns, 0, ns, ns, st);   // u(0) = u(1) = 0
            a.g0 = g;
            a.gout = d_records + (int64_t)g * nt * nch;
            StreamState u{slots, slots + ns, 0, 0};
            launch_stream_steps(dg, a, u, geo.nt - 2, slots, 0, nullptr, nullptr, 0, st);
        }
        NA_CU(cudaGetLastError());
        return TOMO_OK;
    }
    launch_coef(prof, d_f, coef, rcoef, N, cfg->courant, st);
    if (shape.cpl) {
        r.coef = coef;
        r.rcoef = rcoef;
        r.k0 = 1;
        r.T = geo.nt - 2;
        r.ng = geo.G;
        r.cs = shape.cs;
        r.gout = d_records;
        r.nan_on_timeout = true;
        r.w = TileWait{err, 1000000000ull, 0u, nullptr, 0u};   // the contexts' bound, and their variables
        if (const char* v = std::getenv("TOMO_WAIT_LIMIT_NS")) r.w.wait_ns = std::strtoull(v, nullptr, 10);
        if (const char* v = std::getenv("TOMO_TEST_UNDELIVERED_TX")) r.w.extra_tx = (uint32_t)std::strtoul(v, nullptr, 10);
        launch_res_fwd(shape, dg, r, st);
        NA_CU(cudaGetLastError());
        return TOMO_OK;
    }
    // otherwise a group at a time, a step and a gather launch per step
    auto at = [&](int k) { return slots + (int64_t)(k % 3) * N; };
    for (int g = 0; g < geo.G; ++g) {
        launch_zero_slots(slots, 1, 3 * N, 0, N, N, st);   // u(0) = u(1) = 0
        float* const out = d_records + (int64_t)g * nt * nch;
        for (int k = 1; k <= geo.nt - 2; ++k) {
            FwdStep fs{};
            fs.up = at(k - 1);
            fs.uc = at(k);
            fs.un = at(k + 1);
            fs.gstride = 3 * N;
            fs.k = k;
            fs.g0 = g;
            fs.ng = 1;
            launch_fwd_step(prof, dg, coef, rcoef, fs, st);
            GatherStep gs{};
            gs.u = at(k + 1);
            gs.gstride = 3 * N;
            gs.out = out;
            gs.k = k + 1;
            gs.ng = 1;
            launch_gather(dg, gs, st);
        }
    }
    NA_CU(cudaGetLastError());
#undef NA_CU
    return TOMO_OK;
} catch (...) {
    std::string why;
    const tomo_status s = abi_exception(&why);
    std::fprintf(stderr, "tomo_forward_noalloc: %s\n", why.c_str());
    return s;
}
