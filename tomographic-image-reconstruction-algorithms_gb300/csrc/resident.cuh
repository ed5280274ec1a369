// resident.cuh -- sweeps of the benchmark-profile (CFG) physics with the wavefield held on chip.
//
// A thread-block cluster owns one emitter group: its grid rows are cut into bands, one per block,
// and the two wavefield slices of a band live in its threads' registers for the whole sweep.  A
// time step then reads no wavefield from memory: east / west neighbours come from warp shuffles,
// north / south neighbours from the thread's own rows, from rows the block's other warps publish
// in shared memory, and, at a band's edges, from the neighbouring blocks, which write their edge
// row straight into this block's shared memory (st.async) and complete an mbarrier with it.  What
// a step moves through memory is the history the adjoint needs and the records.
//
// Work layout: warp w of a block holds rows RPW w .. RPW w + RPW - 1 of the band; lane l holds
// columns CPL l .. CPL l + CPL - 1 of each, so one warp spans the grid's width (nx <= 32 CPL) and
// cells outside the grid carry zero coefficient and zero sponge factor and stay zero.  Cells are
// evaluated in packed FP32x2 with the operations and rounding of cell.cuh, so a sweep gives the
// bits of the strip and tile kernels.
//
// History.  The forward sweep stores L(k) = Laplacian of u(k), a by-product of its step, and not
// u(k): the adjoint's correlation z(k+1) L(k) is then one read per cell.  History, checkpoints
// and the adjoint state are kept in fragment order -- grid row by grid row, a row as the vectors
// of V consecutive cells [vector in lane][lane] -- so every access of a warp is contiguous whatever
// the width or alignment of the grid.
//
// Measured (one GB300, against the strip and tile kernels on the same grids): 128 x 128, 8 groups:
// 0.35 / 0.40 us per forward / adjoint step (0.83 / 1.18), an iteration of 600 steps 0.58 ms (1.43);
// 256 x 256, one group: 0.42 / 0.62 us (1.2 / 1.6 us in multi-step tiles), an ART iteration of 16
// groups x 2560 steps 55 ms (115.4); 301 x 233, 10 groups (per-cell kernels before): 1.3 / 1.6 us
// (4.2 / 5.6), 2.98 ms per iteration (13.2).  What bounds a step is latency.  ncu, forward sweeps with records:
// 128 x 128, 8 groups on 12 blocks of 11 warps: 91 instructions per warp and step, 2.75 warps per scheduler, 32 %
// of the cycles issue, the block barrier and fixed latencies the largest stalls (2.4 and 1.6 cycles per issue);
// 256 x 256, one group on 16 blocks of 8 warps: 161 instructions, 2 warps per scheduler, 34 % (barrier 1.2, fixed
// latencies 1.2).  DRAM is at 2 to 14 % of its peak.
//
// Waits: only the edge warps wait on other blocks, bounded by TileWait::wait_ns of %globaltimer; a
// wait that runs out sets bit 0 of the host-visible error word and makes the cluster leave.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <type_traits>

#include "bounded_wait.h"
#include "internal.h"

namespace tomo {
namespace {

#include "cell.cuh"
#include "async.cuh"

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Shared-memory address of the same variable in block `rank` of the cluster.
__device__ __forceinline__ uint32_t map_rank(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(a) : "r"(sm_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void st_async2(uint32_t dst, float2 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];\n" ::"r"(dst),
                 "f"(v.x), "f"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async4(uint32_t dst, float2 a, float2 b, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(
                     dst),
                 "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool try_wait_cluster(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// A warp's wait for a neighbour's row, at most limit_ns; the same answer in every lane.
__device__ __forceinline__ bool wait_row(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
    return bounded_wait([&] { return __all_sync(FULL, try_wait_cluster(bar, parity)) != 0; }, [] { return gtimer(); },
                        [&](uint64_t t0) { return __all_sync(FULL, gtimer() - t0 < limit_ns) != 0; });
}

// Geometry of one instantiation.
template <int CPL>
struct Frag {
    static constexpr int NP = CPL / 2;                 // packed pairs per lane and row
    static constexpr int V = CPL % 4 == 0 ? 4 : 2;     // cells per vector
    static constexpr int ROW = 32 * CPL;               // floats per fragment row
    // offset of pair v of a lane in a fragment row
    __device__ __forceinline__ static int at(int lane, int v) {
        return V == 4 ? ((v >> 1) * 32 + lane) * 4 + (v & 1) * 2 : (v * 32 + lane) * 2;
    }
    // offset of grid column x
    __device__ __forceinline__ static int col(int x) {
        const int lane = x / CPL, i = x - lane * CPL;
        return ((i / V) * 32 + lane) * V + i % V;
    }
    __device__ __forceinline__ static void load(float2 (&x)[NP], const float* p, int lane) {
        if constexpr (V == 4) {
#pragma unroll
            for (int v = 0; v < NP; v += 2) {
                const float4 q = *reinterpret_cast<const float4*>(p + at(lane, v));
                x[v] = make_float2(q.x, q.y);
                x[v + 1] = make_float2(q.z, q.w);
            }
        } else {
#pragma unroll
            for (int v = 0; v < NP; ++v) x[v] = *reinterpret_cast<const float2*>(p + at(lane, v));
        }
    }
    __device__ __forceinline__ static void store(float* p, const float2 (&x)[NP], int lane) {
        if constexpr (V == 4) {
#pragma unroll
            for (int v = 0; v < NP; v += 2)
                *reinterpret_cast<float4*>(p + at(lane, v)) = make_float4(x[v].x, x[v].y, x[v + 1].x, x[v + 1].y);
        } else {
#pragma unroll
            for (int v = 0; v < NP; ++v) *reinterpret_cast<float2*>(p + at(lane, v)) = x[v];
        }
    }
    // a row into another block's shared memory, completing its barrier
    __device__ __forceinline__ static void send(uint32_t dst, uint32_t bar, const float2 (&x)[NP], int lane) {
        if constexpr (V == 4) {
#pragma unroll
            for (int v = 0; v < NP; v += 2) st_async4(dst + 4u * at(lane, v), x[v], x[v + 1], bar);
        } else {
#pragma unroll
            for (int v = 0; v < NP; ++v) st_async2(dst + 4u * at(lane, v), x[v], bar);
        }
    }
    // CPL consecutive cells of a natural-order row; zeros from column nx on
    __device__ __forceinline__ static void load_nat(float2 (&x)[NP], const float* row, int lane, int nx, bool ok) {
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            const int i = CPL * lane + 2 * v;
            x[v].x = ok && i < nx ? row[i] : 0.f;
            x[v].y = ok && i + 1 < nx ? row[i + 1] : 0.f;
        }
    }
    __device__ __forceinline__ static void store_nat(float* row, const float2 (&x)[NP], int lane, int nx) {
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            const int i = CPL * lane + 2 * v;
            if (i < nx) row[i] = x[v].x;
            if (i + 1 < nx) row[i + 1] = x[v].y;
        }
    }
};

// Sponge factor of the band's cells: the damp table grows towards the inside, so the factor at the
// nearer of two distances is the smaller of the two factors; 0 outside the grid.
__device__ __forceinline__ float damp1(const DevGeo& g, int i, int n) {
    if (i < 0 || i >= n) return 0.f;
    const int d = min(i, n - 1 - i);
    return d < g.sponge_w ? g.damp[d] : 1.f;
}
__device__ __forceinline__ float2 min2(float2 a, float b) { return make_float2(fminf(a.x, b), fminf(a.y, b)); }

// Laplacian of a lane's two cells u, west and east their outer neighbours: lap5 of cell.cuh.  The
// two-cell sum along the row is scalar (its operands straddle the packed pairs, and packing them
// would cost a move each), the rest packed; every half is rounded as in lap5.
__device__ __forceinline__ float2 row_lap(float west, float2 u, float east, float2 s, float2 n) {
    const float2 ew = make_float2(__fadd_rn(u.y, west), __fadd_rn(east, u.x));
    return pk_fma(make_float2(-4.f, -4.f), u, pk_add(pk_add(ew, s), n));
}
// 2 a - b, rounded once (scalar: the negation is free there)
__device__ __forceinline__ float2 twice_minus(float2 a, float2 b) {
    return make_float2(__fmaf_rn(2.f, a.x, -b.x), __fmaf_rn(2.f, a.y, -b.y));
}

// Shared memory of a block.  The two parities of a row lie next to each other, so a step of known
// parity reaches every row at a constant distance from one running base.
//   bar  [2][2]           rows from the block below (0) and above (1), per parity of the step
//   fail [2], bad         a wait of a pair of steps ran out (by parity of the pair); ... of any
//   halo [2][2][ROW]      [side][parity]: rows received from the neighbouring blocks
//   xch  [W][PR][2][ROW]  rows published per step (PR of each warp's RPW rows)
//   cs   [W RPW][ROW]     coefficient (only where registers do not hold it)
//   ring [D][...]         thread-private prefetch: history rows (adjoint), measured samples (forward)
//   val  [2][nrec]        residuals injected by the next steps (adjoint)
struct ResSmem {
    float *xch, *halo, *cs, *ring, *val;
    uint64_t* bar;
    volatile int *fail, *bad;
};
// Whether a thread's cells are too many to keep the coefficient and sponge factor in registers.
template <int CPL, int RPW>
constexpr bool res_lean_regs = CPL * RPW > 16;
// Steps the adjoint requests its history ahead.
template <int CPL, int RPW>
constexpr int res_depth = CPL * RPW <= 16 ? 4 : CPL * RPW <= 32 ? 2 : 1;
constexpr int RES_MEAS = 8;              // steps the forward sweep requests measured samples ahead

template <int CPL, int RPW, bool FWD>
__host__ __device__ constexpr int res_smem_floats(int W, int part) {   // floats before `part`
    constexpr int ROW = 32 * CPL, PR = FWD ? RPW : RPW < 2 ? 1 : 2;
    const int sizes[4] = {4 * ROW, 2 * W * PR * ROW, CPL * RPW > 16 ? W * RPW * ROW : 0,
                          FWD ? RES_MEAS * 32 * W : res_depth<CPL, RPW> * W * RPW * ROW};
    int n = 0;
    for (int i = 0; i < part; ++i) n += sizes[i];
    return n;
}
template <int CPL, int RPW, bool FWD>
__device__ __forceinline__ ResSmem res_smem(unsigned char* raw, int W) {
    ResSmem s;
    s.bar = reinterpret_cast<uint64_t*>(raw);
    s.fail = reinterpret_cast<volatile int*>(raw + 32);
    s.bad = s.fail + 2;
    float* const f = reinterpret_cast<float*>(raw + 128);
    s.halo = f;
    s.xch = f + res_smem_floats<CPL, RPW, FWD>(W, 1);
    s.cs = f + res_smem_floats<CPL, RPW, FWD>(W, 2);
    s.ring = f + res_smem_floats<CPL, RPW, FWD>(W, 3);
    s.val = f + res_smem_floats<CPL, RPW, FWD>(W, 4);
    return s;
}

// Barriers armed for the first two rows of each side (extra: bytes that never come, for the test of
// the time-out), flags and halo rows cleared.
__device__ __forceinline__ void res_setup(const ResSmem& sm, int rank, int cs, int halo, uint32_t bytes, uint32_t extra) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < 4; ++i) mbar_init(sm.bar + i, 1);
        mbar_fence_init();
        sm.fail[0] = sm.fail[1] = *sm.bad = 0;
        for (int s = 0; s < 2; ++s)
            if (s == 0 ? rank > 0 : rank + 1 < cs)
                for (int p = 0; p < 2; ++p) mbar_expect_tx(sm.bar + 2 * s + p, bytes + extra);
    }
    for (int i = threadIdx.x; i < halo; i += blockDim.x) sm.halo[i] = 0.f;
}

// A block's row links.  Rows are numbered t = 0 (the initial state) .. T; row t has parity t & 1.
// Sending: the edge row goes to the upper halo row of the block below or the lower one of the block
// above and completes that block's barrier.  Receiving, at step t: wait for row t - 1, then arm the
// barrier for row t + 1, which the neighbour sends only once it has this block's row t.  The last
// armed row is never sent (the kernel ends); row T is waited for after the loop.  A wait that runs
// out closes its link in both directions at once: no row is ever sent that is not armed for, which
// would drive the barrier's transaction count below zero (a fault).
template <int CPL>
struct ResLinks {
    uint32_t lo_row, lo_bar, hi_row, hi_bar;   // remote addresses, parity 0
    uint64_t limit_ns;
    bool single = false;                       // the warp's only row is its first
    bool lo, hi;                               // link open: this warp has the block's first / last row, a neighbour beyond
    __device__ __forceinline__ void init(const ResSmem& sm, int rank, int cs, bool first, bool last, uint64_t limit) {
        constexpr int ROW = 32 * CPL;
        lo = first && rank > 0;
        hi = last && rank + 1 < cs;
        limit_ns = limit;
        const uint32_t below = rank > 0 ? rank - 1 : 0, above = rank + 1 < cs ? rank + 1 : rank;
        lo_row = map_rank(sm.halo + 2 * ROW, below);
        lo_bar = map_rank(sm.bar + 2, below);
        hi_row = map_rank(sm.halo, above);
        hi_bar = map_rank(sm.bar, above);
    }
    template <int P>
    __device__ __forceinline__ void send(const float2 (&first)[CPL / 2], const float2 (&last)[CPL / 2], int lane) const {
        constexpr uint32_t step = 4u * 32u * CPL;
        if (lo) Frag<CPL>::send(lo_row + P * step, lo_bar + 8u * P, first, lane);
        if (hi && !single) Frag<CPL>::send(hi_row + P * step, hi_bar + 8u * P, last, lane);
        if (hi && single) Frag<CPL>::send(hi_row + P * step, hi_bar + 8u * P, first, lane);
    }
    // Row t - 1 of parity P.  A wait that runs out is noted for res_failed; the block then leaves.
    template <int P, bool ARM = true>
    __device__ __forceinline__ void recv(const ResSmem& sm, int t, int lane) {
        constexpr uint32_t bytes = 4u * 32u * CPL;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            bool& open = side == 0 ? lo : hi;
            if (!open) continue;
            uint64_t* const b = sm.bar + 2 * side + P;
            if (!wait_row(sm_addr(b), (uint32_t)((t - 1) >> 1) & 1u, limit_ns)) {
                open = false;
                sm.fail[((t - 1) >> 1) & 1] = 1;
                *sm.bad = 1;
            } else if (ARM && lane == 0) {
                mbar_expect_tx(b, bytes);
            }
            __syncwarp();
        }
    }
};
// A failed wait is noted before its step's barrier; every warp reads the note of a pair of steps
// during the next pair (t: its first step) and leaves after it, and the flag is not written again
// before the pair after that, so all warps leave the loop together.
__device__ __forceinline__ int res_failed(const ResSmem& sm, int t) { return sm.fail[(((t - 1) >> 1) & 1) ^ 1]; }

__device__ __forceinline__ void cp_async4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sm_addr(dst)), "l"(__cvta_generic_to_global(src))
                 : "memory");
}
// A thread's cells of one fragment row into its place of a shared-memory row.
template <int CPL>
__device__ __forceinline__ void row_async(float* dst, const float* src, int lane) {
    if constexpr (Frag<CPL>::V == 4) {
#pragma unroll
        for (int v = 0; v < CPL / 2; v += 2) cp_async16(sm_addr(dst + Frag<CPL>::at(lane, v)), src + Frag<CPL>::at(lane, v), true);
    } else {
#pragma unroll
        for (int v = 0; v < CPL / 2; ++v)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sm_addr(dst + Frag<CPL>::at(lane, v))),
                         "l"(__cvta_generic_to_global(src + Frag<CPL>::at(lane, v)))
                         : "memory");
    }
}

// Checkpoints of a forward sweep: chunk ch >= 1 (q from 1 + ch K) restarts from the two slices that
// are newest after a pair of steps: slices ch K and ch K + 1, or, when step ch K + 1 - k0 is a pair's
// first, ch K - 1 and ch K (res_restart tells the recompute which).
__device__ __forceinline__ int restart_slice(int k0, int K, int ch) { return ch * K + 1 - ((ch * K + 1 - k0) & 1); }
// Last step, at least t, of the next pair that ends in a checkpoint (T + 1: none).
__device__ __forceinline__ int res_next_checkpoint(const ResFwd& a, int t) {
    for (int ch = max(1, (a.k0 + t - 1) / a.K); ch < a.nchunk; ++ch) {
        const int e = restart_slice(a.k0, a.K, ch) - a.k0;
        if (e >= t) return e;
    }
    return a.T + 1;
}
// Stores the two newest slices after step t (older, newer) where t ends a checkpoint's pair.
template <int CPL, int RPW>
__device__ __forceinline__ void res_checkpoint(const ResFwd& a, int gl, int64_t fbase, int t, const float2 (&older)[RPW][CPL / 2],
                                               const float2 (&newer)[RPW][CPL / 2], int lane, int rows) {
    const int m = a.k0 + t;
    for (int ch = max(1, m / a.K - 1); ch < a.nchunk && ch * a.K <= m; ++ch) {
        if (restart_slice(a.k0, a.K, ch) != m) continue;
        float* const ck = a.ckpt + gl * a.ckstride + (int64_t)ch * 2 * a.ns + fbase;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            if (r >= rows) continue;
            Frag<CPL>::store(ck + r * Frag<CPL>::ROW, older[r], lane);
            Frag<CPL>::store(ck + a.ns + r * Frag<CPL>::ROW, newer[r], lane);
        }
    }
}

// The records of a group for a caller that cannot be told of a wait that ran out: all NaN.  Called by each block
// with such a wait, behind the cluster's last barrier and so after every block's records (a block can finish on
// rows computed past a neighbour's failed wait: the whole group is given up).  It stands in the failed branch and
// reads the group's number again: behind the common path it cost the steps of one row per warp 2 to 5 %
// (256 x 256, one group at a time: 59.9 -> 62.8 ms an iteration; as a launch of its own 5 us a call).
__device__ __forceinline__ void res_nan_records(float* gout, int64_t n) {
    uint32_t gl;
    asm volatile("mov.u32 %0, %%clusterid.x;\n" : "=r"(gl));
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) gout[gl * n + i] = __int_as_float(0x7fffffff);
}

// ---------------------------------------------------------------------------------------------
// Forward sweep: slices k0+1 .. k0+T of every group of the launch.
//
// A step's chain is short (two shared-memory reads, two shuffles, seven dependent operations, one
// write, one barrier), so on small grids what a step costs is every instruction around that chain.
// The steps therefore run as two loops over pairs of steps: one for the steps that add a source,
// and a plain one with running pointers, whose only tests are the warp-uniform edge and record
// tests and, per pair, the checkpoint and time-out tests.
template <int CPL, int RPW, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_res_fwd(DevGeo g, ResFwd a) {
    using F = Frag<CPL>;
    constexpr int NP = F::NP, ROW = F::ROW;
    constexpr bool CS = res_lean_regs<CPL, RPW>;
    extern __shared__ __align__(1024) unsigned char smraw[];
    // w through a shuffle: the compiler then knows it is the same for the whole warp and its tests branch uniformly
    const int W = blockDim.x >> 5, lane = threadIdx.x & 31, w = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);
    const ResSmem sm = res_smem<CPL, RPW, true>(smraw, W);
    const int rank = (int)cluster_rank(), cs = a.cs, gl = blockIdx.x / cs;
    const int RB = W * RPW, jb = rank * RB, jw = jb + w * RPW;
    const int nx = g.nx, ny = g.ny, ggl = a.g0 + gl, T = a.T;
    res_setup(sm, rank, cs, 4 * ROW, 4u * ROW, a.w.extra_tx);
    ResLinks<CPL> lk;
    lk.init(sm, rank, cs, w == 0, w == W - 1, a.w.wait_ns);
    const int64_t fbase = (int64_t)jw * ROW;
    // coefficient, sponge factors (the product rule of damp1 where registers are short), state
    float2 cc[CS ? 1 : RPW][NP], dd[CS ? 1 : RPW][NP], ua[RPW][NP], ub[RPW][NP];
    float drow[RPW];
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int j = jw + r;
        drow[r] = damp1(g, j, ny);
        float2 t[NP];
        F::load_nat(t, a.coef + (int64_t)j * nx, lane, nx, j < ny);
        if constexpr (CS) F::store(sm.cs + (w * RPW + r) * ROW, t, lane);
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            ua[r][v] = ub[r][v] = make_float2(0.f, 0.f);   // u(k0), u(k0-1)
            if (!CS || r == 0) {
                const float2 d = make_float2(damp1(g, CPL * lane + 2 * v, nx), damp1(g, CPL * lane + 2 * v + 1, nx));
                cc[CS ? 0 : r][v] = t[v];
                dd[CS ? 0 : r][v] = CS ? d : min2(d, drow[r]);
            }
        }
        if (a.in0 && j < ny) {
            F::load(ub[r], a.in0 + gl * a.instride + (int64_t)j * ROW, lane);
            F::load(ua[r], a.in1 + gl * a.instride + (int64_t)j * ROW, lane);
        }
    }
    // this thread's receiver (the block's receivers are consecutive in row order, dealt out from the second
    // warp on: the first and the last have the links to attend to)
    const int n0 = a.gout ? a.rowstart[min(jb, ny)] : 0, n1 = a.gout ? a.rowstart[min(jb + RB, ny)] : 0;
    const bool noisy = a.gmeas && g.noise_key;
    const uint64_t key = noisy ? *g.noise_key : 0;
    const int64_t rbase = (int64_t)gl * g.nt * g.nch;
    int roff = 0, rch = 0;
    const int ri = 32 * ((w + W - 1) % W) + lane;
    const bool rec = n0 + ri < n1, rec_more = n0 + (int)blockDim.x < n1;
    if (rec) {
        const int q = a.rcell[n0 + ri], j = q / nx;
        roff = (j - jb) * 2 * ROW + F::col(q - j * nx);
        rch = a.rchan[n0 + ri];
    }
    const bool rec_warp = n0 + ri - lane < n1, meas = rec && a.gmeas;
    float* op = rec ? a.gout + rbase + (int64_t)(a.k0 + 1) * g.nch + rch : nullptr;         // slice k0 + 1
    const float* mp = meas ? a.gmeas + rbase + (int64_t)(a.k0 + 1) * g.nch + rch : nullptr;
    const float* const pub0 = sm.xch + roff;
    float* const mring = sm.ring + threadIdx.x;
    int mi = 0, mleft = meas ? T : 0;                    // slices k0+1 .. k0+T still to request
    auto request = [&](int i) {                          // the next measured sample into place i
        if (mleft > 0) {
            cp_async4(mring + i * 32 * W, mp);
            mp += g.nch;
            --mleft;
        }
        cp_async_commit();
    };
    auto put = [&](float v, float mv, float* o, int m, int ch) {
        if (noisy) v = v * noise_factor(key, g.noise_level, ggl, m, ch);
        *o = a.gmeas ? mv - v : v;
    };
    // records of slice m from the rows published with parity P
    auto record = [&](int m, auto pc) {
        constexpr int P = decltype(pc)::value;
        if (rec_warp && rec) {
            float mv = 0.f;
            if (meas) {
                cp_async_wait<RES_MEAS - 1>();
                mv = mring[mi * 32 * W];
                request(mi);
                mi = mi + 1 == RES_MEAS ? 0 : mi + 1;
            }
            put(pub0[P * ROW], mv, op, m, rch);
            op += g.nch;
        }
        if (rec_more) {
            for (int n = n0 + ri + blockDim.x; n < n1; n += blockDim.x) {
                const int q = a.rcell[n], j = q / nx, ch = a.rchan[n];
                const int64_t o = rbase + (int64_t)m * g.nch + ch;
                put(sm.xch[((j - jb) * 2 + P) * ROW + F::col(q - j * nx)], a.gmeas ? a.gmeas[o] : 0.f, a.gout + o, m, ch);
            }
        }
    };
    float* const xw = sm.xch + w * RPW * 2 * ROW;
    auto publish = [&](const float2 (&x)[RPW][NP], auto pc) {
        constexpr int P = decltype(pc)::value;
#pragma unroll
        for (int r = 0; r < RPW; ++r) F::store(xw + (r * 2 + P) * ROW, x[r], lane);
        lk.template send<P>(x[0], x[RPW - 1], lane);
    };
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;
    if (meas)
        for (int i = 0; i < RES_MEAS; ++i) request(i);
    __syncthreads();
    cluster_sync();            // every block's barriers are armed and its halo rows cleared
    publish(ua, P0{});
    __syncthreads();

    const float* const srow = w > 0 ? xw - 2 * ROW : sm.halo;                          // parity 0
    const float* const nrow = w < W - 1 ? xw + RPW * 2 * ROW : sm.halo + 2 * ROW;
    const int tkeep = a.hist ? a.qlo - a.k0 + 1 : T + 1;   // steps t >= tkeep store L(k0 + t - 1)
    float* hp = a.hist ? a.hist + gl * a.hstride + fbase : nullptr;
    // one step: u(m) from cur = u(m-1) and prv = u(m-2), written over prv; the rows of u(m-1) were
    // published with parity P.  SRC: the source src is added to the cells of em.
    auto step = [&](float2 (&cur)[RPW][NP], float2 (&prv)[RPW][NP], int t, auto pc, auto src_c, float src,
                    const unsigned* em) {
        constexpr int P = decltype(pc)::value;
        constexpr bool SRC = decltype(src_c)::value;
        lk.template recv<P>(sm, t, lane);
        float2 sb[NP], nb[NP];
        F::load(sb, srow + P * ROW, lane);
        F::load(nb, nrow + P * ROW, lane);
        const bool keep = t >= tkeep;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            float wl = __shfl_up_sync(FULL, cur[r][NP - 1].y, 1), er = __shfl_down_sync(FULL, cur[r][0].x, 1);
            wl = lane == 0 ? 0.f : wl;
            er = lane == 31 ? 0.f : er;
            float2 lap[NP], cr[NP];
            if constexpr (CS) F::load(cr, sm.cs + (w * RPW + r) * ROW, lane);
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                const float2 u = cur[r][v];
                const float2 s = r == 0 ? sb[v] : cur[r - 1][v], n = r == RPW - 1 ? nb[v] : cur[r + 1][v];
                lap[v] = row_lap(v > 0 ? cur[r][v - 1].y : wl, u, v + 1 < NP ? cur[r][v + 1].x : er, s, n);
                const float2 c = CS ? cr[v] : cc[CS ? 0 : r][v];
                const float2 d = CS ? min2(dd[0][v], drow[r]) : dd[CS ? 0 : r][v];
                const float2 x = pk_fma(c, lap[v], twice_minus(u, prv[r][v]));
                if constexpr (SRC) {
                    const float2 am = make_float2((em[r] >> (2 * v)) & 1u ? src : 0.f, (em[r] >> (2 * v)) & 2u ? src : 0.f);
                    prv[r][v] = pk_fma(d, x, am);
                } else {
                    prv[r][v] = pk_mul(d, x);
                }
            }
            if (keep && jw + r < ny) F::store(hp + r * ROW, lap, lane);
        }
        publish(prv, std::integral_constant<int, (P ^ 1)>{});
        if (keep) hp += a.ns;
    };
    int t = 1;
    bool live = true;
    {
        // steps with a source, and the first pair (slice k0 is not recorded)
        unsigned em[RPW];
#pragma unroll
        for (int r = 0; r < RPW; ++r) em[r] = 0u;
        if (a.k0 < g.n_src_steps)
            for (int e = 0; e < g.gs; ++e) {
                const int q = g.emit[(int64_t)ggl * g.gs + e], j = q / nx, x = q - j * nx;
#pragma unroll
                for (int r = 0; r < RPW; ++r)
                    if (j == jw + r && x / CPL == lane) em[r] |= 1u << (x % CPL);
            }
        const int tsrc = max(1, min(T, g.n_src_steps - a.k0));
#pragma unroll 1
        for (; t <= tsrc && live; t += 2) {
            const int k = a.k0 + t - 1, failed = res_failed(sm, t);
            step(ua, ub, t, P0{}, std::true_type{}, k < g.n_src_steps ? g.src[k] : 0.f, em);
            if (t > 1) record(k, P0{});
            __syncthreads();
            if (t < T) {
                step(ub, ua, t + 1, P1{}, std::true_type{}, k + 1 < g.n_src_steps ? g.src[k + 1] : 0.f, em);
                record(k + 1, P1{});
                __syncthreads();
            }
            live = failed == 0;
            if (a.ckpt && t + 1 <= T) res_checkpoint<CPL, RPW>(a, gl, fbase, t + 1, ub, ua, lane, ny - jw);
        }
    }
    // pairs of plain steps; tck: the pair's last step after which the two newest slices are a checkpoint
    int tck = a.ckpt ? res_next_checkpoint(a, t) : T + 1;
#pragma unroll 1
    for (; t + 1 <= T && live; t += 2) {
        const int failed = res_failed(sm, t);
        step(ua, ub, t, P0{}, std::false_type{}, 0.f, nullptr);
        record(a.k0 + t - 1, P0{});
        __syncthreads();
        step(ub, ua, t + 1, P1{}, std::false_type{}, 0.f, nullptr);
        record(a.k0 + t, P1{});
        __syncthreads();
        live = failed == 0;
        if (t + 1 == tck) {
            res_checkpoint<CPL, RPW>(a, gl, fbase, t + 1, ub, ua, lane, ny - jw);
            tck = res_next_checkpoint(a, t + 2);
        }
    }
    if (t == T && live) {
        step(ua, ub, t, P0{}, std::false_type{}, 0.f, nullptr);
        record(a.k0 + t - 1, P0{});
        __syncthreads();
    }
    // the neighbours' rows T: nothing is in flight towards this block afterwards
    if (live) {
        if (T & 1) lk.template recv<1, false>(sm, T + 1, lane);
        else lk.template recv<0, false>(sm, T + 1, lane);
    }
    __syncthreads();
    if (*sm.bad == 0) {
        if (T & 1) record(a.k0 + T, P1{});
        else record(a.k0 + T, P0{});
        if (a.out) {
#pragma unroll
            for (int r = 0; r < RPW; ++r)
                if (jw + r < ny) {
                    float* o = a.out + gl * a.outstride + (int64_t)(jw + r) * nx;
                    if (T & 1) F::store_nat(o, ub[r], lane, nx);
                    else F::store_nat(o, ua[r], lane, nx);
                }
        }
    } else {
        if (threadIdx.x == 0) atomicOr(a.w.err, 1u);
        if (a.nan_on_timeout) {
            cp_async_wait<0>();
            cluster_sync();
            res_nan_records(a.gout, (int64_t)g.nt * g.nch);
            return;
        }
    }
    cp_async_wait<0>();
    cluster_sync();            // no block leaves while another may still write its shared memory
}

// ---------------------------------------------------------------------------------------------
// Adjoint sweep with the residual injection and the correlation: z(kz0) .. z(kz0-T+1).  State
// (z(kz0+1), z(kz0+2), correlation) in fragment order at a.st, slices a.ns apart: zero when a.first;
// the last launch of a sweep (a.last) writes the correlation in natural order instead.  The
// history is requested res_depth steps ahead by thread-private asynchronous copies.
template <int CPL, int RPW, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_res_adj(DevGeo g, ResAdj a) {
    using F = Frag<CPL>;
    constexpr int NP = F::NP, ROW = F::ROW, PR = RPW < 2 ? 1 : 2, D = res_depth<CPL, RPW>;
    constexpr bool CS = res_lean_regs<CPL, RPW>, EARLY = CPL * RPW <= 8;
    extern __shared__ __align__(1024) unsigned char smraw[];
    // w through a shuffle: the compiler then knows it is the same for the whole warp and its tests branch uniformly
    const int W = blockDim.x >> 5, lane = threadIdx.x & 31, w = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);
    const ResSmem sm = res_smem<CPL, RPW, false>(smraw, W);
    const int rank = (int)cluster_rank(), cs = a.cs, gl = blockIdx.x / cs;
    const int RB = W * RPW, jb = rank * RB, jw = jb + w * RPW;
    const int nx = g.nx, ny = g.ny, T = a.T;
    res_setup(sm, rank, cs, 4 * ROW, 4u * ROW, a.w.extra_tx);
    ResLinks<CPL> lk;
    lk.init(sm, rank, cs, w == 0, w == W - 1, a.w.wait_ns);
    const int64_t fbase = (int64_t)jw * ROW;
    // history of the first D steps
    const float* hp = a.hist + gl * a.hstride + (int64_t)(a.kz0 - 1 - a.qlo) * a.ns + fbase;
    float* const ring = sm.ring + w * RPW * ROW;
    int left = T;                                        // steps whose history is still to request
    auto request = [&](int i) {
        if (left > 0) {
#pragma unroll
            for (int r = 0; r < RPW; ++r)
                if (jw + r < ny) row_async<CPL>(ring + (i * RB + r) * ROW, hp + r * ROW, lane);
            hp -= a.ns;
            --left;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int r = 0; r < RPW; ++r)                        // rows below the grid are never requested
        if (jw + r >= ny) {
            const float2 none[NP] = {};
            for (int i = 0; i < D; ++i) F::store(ring + (i * RB + r) * ROW, none, lane);
        }
    for (int i = 0; i < D; ++i) request(i);
    float2 cc[CS ? 1 : RPW][NP], dd[CS ? 1 : RPW][NP], za[RPW][NP], zb[RPW][NP], pa[RPW][NP], pb[RPW][NP], co[RPW][NP];
    float drow[RPW];
    unsigned rm[RPW];          // receivers among the thread's cells of row r
    int rb[RPW];               // index of the first of them in the block's receivers
    const int n0 = a.rowstart[min(jb, ny)], n1 = a.rowstart[min(jb + RB, ny)], nrec = n1 - n0;
    const float2 zero = make_float2(0.f, 0.f);
    float* const st = a.st + gl * a.ststride + fbase;
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int j = jw + r;
        drow[r] = damp1(g, j, ny);
        float2 c[NP];
        F::load_nat(c, a.coef + (int64_t)j * nx, lane, nx, j < ny);
        if constexpr (CS) F::store(sm.cs + (w * RPW + r) * ROW, c, lane);
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            za[r][v] = zb[r][v] = co[r][v] = zero;
            if (!CS || r == 0) {
                const float2 d = make_float2(damp1(g, CPL * lane + 2 * v, nx), damp1(g, CPL * lane + 2 * v + 1, nx));
                cc[CS ? 0 : r][v] = c[v];
                dd[CS ? 0 : r][v] = CS ? d : min2(d, drow[r]);
            }
        }
        if (!a.first && j < ny) {
            F::load(za[r], st + r * ROW, lane);
            F::load(zb[r], st + a.ns + r * ROW, lane);
            F::load(co[r], st + 2 * a.ns + r * ROW, lane);
        }
#pragma unroll
        for (int v = 0; v < NP; ++v) pa[r][v] = pk_mul(c[v], za[r][v]);
        rm[r] = 0u;
        rb[r] = 0;
        if (j < ny)
            for (int n = a.rowstart[j]; n < a.rowstart[j + 1]; ++n) {
                const int x = a.rcell[n] - j * nx;
                if (x / CPL == lane) {
                    if (!rm[r]) rb[r] = n - n0;
                    rm[r] |= 1u << (x % CPL);
                }
            }
    }
    unsigned row_rcv = 0u;     // bit r: some lane holds a receiver of row r
#pragma unroll
    for (int r = 0; r < RPW; ++r) row_rcv |= __any_sync(FULL, rm[r] != 0u) ? 1u << r : 0u;
    // this thread's share of the residual staging: one receiver (and, rarely, every blockDim-th
    // more); step t's residuals lie in val[t & 1], staged a step before from a register loaded two
    // steps before that
    const float* const rr = a.rr + gl * a.rrstride;
    const int ri = 32 * ((w + W - 1) % W) + lane;
    const bool stg = ri < nrec, stg_more = (int)blockDim.x < nrec;
    const float* rp = stg ? rr + (int64_t)a.kz0 * g.nch + a.rchan[n0 + ri] : nullptr;
    int rleft = stg ? T : 0;
    auto next_res = [&](float& v) {
        if (rleft > 0) {
            v = *rp;
            rp -= g.nch;
            --rleft;
        }
    };
    auto stage = [&](int t, auto pc, float v) {
        constexpr int P = decltype(pc)::value;
        if (stg) sm.val[P * nrec + ri] = v;
        if (stg_more && t <= T)
            for (int n = ri + blockDim.x; n < nrec; n += blockDim.x)
                sm.val[P * nrec + n] = rr[(int64_t)(a.kz0 - t + 1) * g.nch + a.rchan[n0 + n]];
    };
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;
    float rv0 = 0.f, rv1 = 0.f;                          // residuals of the next even / odd step to stage
    next_res(rv1);
    stage(1, P1{}, rv1);
    next_res(rv0);
    next_res(rv1);
    float* const xw = sm.xch + w * PR * 2 * ROW;
    auto publish = [&](const float2 (&x)[RPW][NP], auto pc) {
        constexpr int P = decltype(pc)::value;
        F::store(xw + P * ROW, x[0], lane);
        if constexpr (PR > 1) F::store(xw + (2 + P) * ROW, x[RPW - 1], lane);
        lk.template send<P>(x[0], x[RPW - 1], lane);
    };
    __syncthreads();
    cluster_sync();
    publish(pa, P0{});
    __syncthreads();

    const float* const srow = w > 0 ? xw - 2 * ROW : sm.halo;
    const float* const nrow = w < W - 1 ? xw + PR * 2 * ROW : sm.halo + 2 * ROW;
    int hi = 0;
    // one step: z(m) from zc = z(m+1) (products pc) and zp = z(m+2), written over zp, its products over pn
    auto step = [&](float2 (&zc)[RPW][NP], float2 (&zp)[RPW][NP], float2 (&pc)[RPW][NP], float2 (&pn)[RPW][NP], int t,
                    auto par) {
        constexpr int P = decltype(par)::value;
        lk.template recv<P>(sm, t, lane);
        const float* const vals = sm.val + (P ^ 1) * nrec;
        float2 sb[NP], nb[NP];
        F::load(sb, srow + P * ROW, lane);
        F::load(nb, nrow + P * ROW, lane);
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            float wl = __shfl_up_sync(FULL, pc[r][NP - 1].y, 1), er = __shfl_down_sync(FULL, pc[r][0].x, 1);
            wl = lane == 0 ? 0.f : wl;
            er = lane == 31 ? 0.f : er;
            float2 cr[NP];
            if constexpr (CS) F::load(cr, sm.cs + (w * RPW + r) * ROW, lane);
            // residuals of the row's receivers: small tiles, whose step is one dependent chain, load them
            // ahead of it and always add; large ones add to the cells that have one, in such rows only
            float2 x[NP], inj[EARLY ? NP : 1];
            if constexpr (EARLY) {
#pragma unroll
                for (int v = 0; v < NP; ++v) inj[v] = zero;
                if ((row_rcv >> r) & 1u) {
                    int b = rb[r];
#pragma unroll
                    for (int v = 0; v < NP; ++v) {
                        if ((rm[r] >> (2 * v)) & 1u) inj[v].x = vals[b++];
                        if ((rm[r] >> (2 * v)) & 2u) inj[v].y = vals[b++];
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                const float2 q = pc[r][v];
                const float2 s = r == 0 ? sb[v] : pc[r - 1][v], n = r == RPW - 1 ? nb[v] : pc[r + 1][v];
                const float2 lz = row_lap(v > 0 ? pc[r][v - 1].y : wl, q, v + 1 < NP ? pc[r][v + 1].x : er, s, n);
                x[v] = pk_add(twice_minus(zc[r][v], zp[r][v]), lz);
                if constexpr (EARLY) x[v] = pk_add(x[v], inj[v]);
            }
            if (!EARLY && ((row_rcv >> r) & 1u)) {
                int b = rb[r];
#pragma unroll
                for (int v = 0; v < NP; ++v) {
                    if ((rm[r] >> (2 * v)) & 1u) x[v].x = __fadd_rn(x[v].x, vals[b++]);
                    if ((rm[r] >> (2 * v)) & 2u) x[v].y = __fadd_rn(x[v].y, vals[b++]);
                }
            }
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                zp[r][v] = pk_mul(CS ? min2(dd[0][v], drow[r]) : dd[CS ? 0 : r][v], x[v]);
                pn[r][v] = pk_mul(CS ? cr[v] : cc[CS ? 0 : r][v], zp[r][v]);
            }
        }
        publish(pn, std::integral_constant<int, (P ^ 1)>{});
        if constexpr (P == 0) {
            stage(t + 1, P0{}, rv0);
            next_res(rv0);
        } else {
            stage(t + 1, P1{}, rv1);
            next_res(rv1);
        }
        cp_async_wait<D - 1>();
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            float2 lu[NP];
            F::load(lu, ring + (hi * RB + r) * ROW, lane);
#pragma unroll
            for (int v = 0; v < NP; ++v) co[r][v] = pk_fma(zp[r][v], lu[v], co[r][v]);
        }
        request(hi);
        if (D > 1) hi = hi + 1 == D ? 0 : hi + 1;
        __syncthreads();
    };
    bool live = true;
#pragma unroll 1
    for (int t = 1; t <= T && live; t += 2) {
        const int failed = res_failed(sm, t);
        step(za, zb, pa, pb, t, P0{});                   // z(kz0-t+1) into zb
        if (t == T) break;
        step(zb, za, pb, pa, t + 1, P1{});               // z(kz0-t) into za
        live = failed == 0;
    }
    if (live) {
        if (T & 1) lk.template recv<1, false>(sm, T + 1, lane);
        else lk.template recv<0, false>(sm, T + 1, lane);
    }
    __syncthreads();
    if (*sm.bad == 0) {
        const bool odd = T & 1;                          // odd T: the newest slice is in zb
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            if (jw + r >= ny) continue;
            if (a.last) {
                F::store_nat(a.corr + gl * a.cstride + (int64_t)(jw + r) * nx, co[r], lane, nx);
            } else {
#pragma unroll
                for (int v = 0; v < NP; ++v) {
                    const float2 x = za[r][v], y = zb[r][v];
                    za[r][v] = odd ? y : x;
                    zb[r][v] = odd ? x : y;
                }
                F::store(st + r * ROW, za[r], lane);
                F::store(st + a.ns + r * ROW, zb[r], lane);
                F::store(st + 2 * a.ns + r * ROW, co[r], lane);
            }
        }
    } else if (threadIdx.x == 0) {
        atomicOr(a.w.err, 1u);
    }
    cp_async_wait<0>();
    cluster_sync();
}

// ---- host side of one width -----------------------------------------------------------------
template <int CPL, int RPW>
size_t res_smem_bytes(int W, bool fwd, int nrec) {
    return 128 + 4 * (fwd ? (size_t)res_smem_floats<CPL, RPW, true>(W, 4)
                          : (size_t)res_smem_floats<CPL, RPW, false>(W, 4) + 2 * (size_t)nrec);
}

inline void res_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr, const ResShape& s, int ng, size_t smem,
                       void* stream) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)(s.cs * ng));
    cfg.blockDim = dim3((unsigned)(32 * s.warps));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = (cudaStream_t)stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s.cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

// Prepares a kernel for clusters of up to 16 blocks and the shared memory of its largest block.
template <typename Kern>
bool res_prepare(Kern kern) {
    int dev = 0, cap = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return false;
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cap) == cudaSuccess &&
           cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
}

// Runs one instantiation: a launch (args set), or the count of clusters the GPU holds at once.
template <typename Kern, typename Args>
cudaError_t res_call(Kern kern, const ResShape& s, size_t smem, const DevGeo* g, const Args* a, int* held, void* stream) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    res_config(cfg, attr, s, a ? a->ng : 1, smem, stream);
    if (!res_prepare(kern)) return cudaErrorInvalidValue;
    if (held) return cudaOccupancyMaxActiveClusters(held, reinterpret_cast<const void*>(kern), &cfg);
    return cudaLaunchKernelEx(&cfg, kern, *g, *a);
}

// Up to 8 warps a thread may use 255 registers, up to 16 warps 128 (the wider thread tiles need more).
template <int CPL, int RPW, typename Args>
cudaError_t res_go(const ResShape& s, const DevGeo* g, const Args* a, int* held, void* stream) {
    constexpr bool fwd = std::is_same<Args, ResFwd>::value;
    const size_t smem = res_smem_bytes<CPL, RPW>(s.warps, fwd, s.nrec);
    if (s.warps > 8) {
        if constexpr (CPL * RPW <= 16) {
            if constexpr (fwd) return res_call(k_res_fwd<CPL, RPW, 512>, s, smem, g, a, held, stream);
            else return res_call(k_res_adj<CPL, RPW, 512>, s, smem, g, a, held, stream);
        } else {
            return cudaErrorInvalidValue;
        }
    }
    if constexpr (fwd) return res_call(k_res_fwd<CPL, RPW, 256>, s, smem, g, a, held, stream);
    else return res_call(k_res_adj<CPL, RPW, 256>, s, smem, g, a, held, stream);
}

}  // namespace
}  // namespace tomo
