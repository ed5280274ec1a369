// stream.cu -- several time steps per launch on grids that do not fit on chip (CFG physics).
//
// A warp carries a strip of columns down a band of rows with T time levels in flight: at row j it
// loads the two input slices, computes the first level at row j - 1, the second at row j - 2, .. the
// T-th at row j - T.  The rows a level needs of the one before it are in registers, so the slices
// between the first and the last level never touch memory: a launch reads two slices and writes two
// per T steps (one each for T = 1), plus the history the adjoint needs.  As in the resident sweeps the history
// is L(k) = Laplacian of u(k), a by-product of the forward step, which the adjoint reads once per cell.
//
// What bounds it: bytes.  The per-step kernels move 4 (forward) and 6 (adjoint) slices per step and group;
// with T = 4 a step moves 1 (2 with the history) and 2.5, times the halo's share below.  Measured, us per
// step, per-step kernels -> this: 32 groups of 512 x 512 forward 14.9 -> 9.4 (with history 14.1), adjoint
// 27.5 -> 21.8; 8 of 2048 x 2048 forward 55.8 -> 27.5 (51.6), adjoint 96 -> 74 (4.5 of 6.8 TB/s in
// the last two, halo rows not counted).  Iterations of these problems: 134.4 -> 119.9 ms with 256 receivers
// and checkpoints every 50 steps, 77.1 -> 55.9 ms.  Four levels because eight need registers for 24 rows
// and a halo of 8 on each side.
//
// Halo.  Strips overlap by 8 columns on each side in the forward sweep, whose lanes hold 4 cells (128
// columns, 112 owned), and by 4 in the adjoint, whose lanes hold 2 (64 columns, 56 owned: its levels need
// twice the registers); bands overlap by T <= 4 rows; both are computed twice.  Slices carry a frame of
// guard cells (STREAM_TOP rows above, STREAM_BOTTOM below, STREAM_LEFT columns on either side of whole
// 32-byte sectors; pitch px), so no access of the row loop tests a bound: guard cells have zero coefficient
// and sponge factor, stay zero, and keep whatever lies beyond them out of the grid.
//
// Inputs arrive by asynchronous copies of 16 bytes, six rows ahead in the forward sweep and three in the
// adjoint; the row loop is unrolled by three, so that the rolling rows and the ring slots are fixed names.
// The coefficient of a row (and, in the adjoint, its sponge factor) stays in the ring until the last level has
// passed it; the forward sweep takes the sponge factor from its row and column.
//
// Records: the forward launch writes simulated samples; k_resid_meas turns them into residuals
// afterwards, so no level waits for a measured sample.  The adjoint's residuals at the receivers of a
// warp's strip are staged in shared memory before its row loop.
//
// Same cell arithmetic, operand order and rounding as cell.cuh: same bits as the per-step kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "internal.h"

namespace tomo {
namespace {

#include "cell.cuh"

constexpr int SW = 4;            // warps per block
constexpr int FH = 8, AH = 4;    // columns of overlap on each side: forward (whole sectors), adjoint
constexpr int FW = 128, FOWN = FW - 2 * FH;     // forward strip: columns, owned columns
constexpr int AW = 64, AOWN = AW - 2 * AH;      // adjoint strip
constexpr int MAXR = 128;        // rows of a band at most
constexpr int FD = 6, FC = 12;   // forward ring slots: slices, coefficient (groups of 3)
constexpr int AD = 3, AC = 9;    // adjoint ring slots
constexpr int NREC = 128;        // receivers of a warp's strip kept in shared memory

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp16(uint32_t dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(saddr(dst)), "l"(src) : "memory");
}
// ((e + w) + s) + n - 4 u of two cells; the sum along the row is scalar (see resident.cuh)
__device__ __forceinline__ float2 lap_row(float west, float2 u, float east, float2 s, float2 n) {
    const float2 ew = make_float2(__fadd_rn(u.y, west), __fadd_rn(east, u.x));
    return pk_fma(make_float2(-4.f, -4.f), u, pk_add(pk_add(ew, s), n));
}
__device__ __forceinline__ float2 twice_less(float2 a, float2 b) {
    return make_float2(__fmaf_rn(2.f, a.x, -b.x), __fmaf_rn(2.f, a.y, -b.y));
}

// Sponge factor of a column or a row (0 outside the grid).
__device__ __forceinline__ float damp_line(const DevGeo& g, int k, int n) {
    if (k < 0 || k >= n) return 0.f;
    const int d = min(k, n - 1 - k);
    return d < g.sponge_w ? g.damp[d] : 1.f;
}
__device__ __forceinline__ float damp_col(const DevGeo& g, int x) { return damp_line(g, x, g.nx); }
__device__ __forceinline__ float damp_row(const DevGeo& g, int y) { return damp_line(g, y, g.ny); }

// Receivers of rows ya .. yb-1 and columns [xa, xb) in a warp's shared memory: per row the index of
// the first and the count, per receiver its column from x0 (low byte) and its channel, so the row loop does not
// wait for the global tables (launches of four steps that write records, 32 groups of 512 x 512: 57 -> 49 us,
// the adjoint's 87 -> 83).  Returns their number (may exceed NREC: the rows beyond are found in the global tables).
struct RowRec {
    uint16_t first;
    uint16_t count;
};
__device__ __forceinline__ int list_receivers(const StreamRec& t, int ny, int ya, int yb, int x0, int xa, int xb, int nx, RowRec* rows,
                                              int* ent, int lane) {
    for (int y = ya + lane; y < yb; y += 32) rows[y - ya] = RowRec{0, 0};
    const int e0 = t.rowstart[max(ya, 0)], e1 = t.rowstart[min(yb, ny)];
    __syncwarp();
    int total = 0;
    for (int e = e0; e < e1; e += 32) {                    // the rows' receivers, 32 at a time (a lane to each
                                                           // row waits for a chain of loads along the ring's top)
        const int q = e + lane < e1 ? t.rcell[e + lane] : -1, r = q / nx, x = q - r * nx;
        const bool in = q >= 0 && x >= xa && x < xb;
        const unsigned b = __ballot_sync(FULL, in), same = __match_any_sync(FULL, in ? r : -1);
        const int at = total + __popc(b & ((1u << lane) - 1u));
        if (in) {
            if (at < NREC) ent[at] = (x - x0) | t.rchan[e + lane] << 8;
            if ((same & ((1u << lane) - 1u)) == 0u) {      // the row's first of these
                RowRec& row = rows[r - ya];
                if (row.count == 0) row.first = (uint16_t)min(at, 65535);
                row.count += (uint16_t)__popc(same);
            }
        }
        total += __popc(b);
        __syncwarp();
    }
    return total;
}

// ---------------------------------------------------------------------------------------------
// Forward: slices k0+1 .. k0+T.
template <int T, bool SRC>
__global__ void __launch_bounds__(SW * 32, 4) k_stream_fwd(DevGeo g, StreamFwd a) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, w = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);
    const int ny = g.ny, px = a.px;
    // warps are dealt out over (group, band, strip), the strip running fastest
    const int id = blockIdx.x * SW + w, strip = id % a.strips, gl = id / a.bands / a.strips;
    const int x0 = strip * FOWN - FH, i = x0 + 4 * lane;
    const int y0 = id / a.strips % a.bands * a.R, yend = min(y0 + a.R, ny);
    // per warp: u, v [FD][FW]; c [FC][FW]; receivers; sponge factor of each row
    constexpr int WF = (2 * FD + FC) * FW;
    float* const base = reinterpret_cast<float*>(smem4) + w * (WF + 2 * MAXR + 16 + NREC);
    float* const ru = base + 4 * lane;                     // this lane's places
    constexpr int V = FD * FW, C = 2 * FD * FW;            // from u: v, c
    RowRec* const rows = reinterpret_cast<RowRec*>(base + WF);
    int* const ent = reinterpret_cast<int*>(base + WF + MAXR);
    float* const drow = base + WF + MAXR + NREC;       // of row ja + t
    if (gl >= a.ng) return;
    const bool own = i >= 0 && i < g.nx && lane >= FH / 4 && lane < (FW - FH) / 4;
    const float* const u0 = a.in1 + gl * a.in1stride;
    const float* const v0 = a.in0 + gl * a.in0stride - px;  // row j - 1 at row j's offset
    float* const o1 = a.out1 + gl * a.outstride;
    float* const o0 = T > 1 ? a.out0 + gl * a.outstride : nullptr;
    float* const hist = a.hist ? a.hist + gl * a.hstride + (int64_t)(a.k0 - a.qlo) * a.ns : nullptr;
    float* const gout = a.gout ? a.gout + ((int64_t)gl * g.nt + a.k0) * g.nch : nullptr;
    float src[T];
#pragma unroll
    for (int s = 0; s < T; ++s) src[s] = SRC && a.k0 + s < g.n_src_steps ? g.src[a.k0 + s] : 0.f;
    const int32_t* const em = g.emit + (int64_t)(a.g0 + gl) * g.gs;
    const int ja = y0 - T, jn = yend - y0 + 2 * T;         // iterations j = ja + t, t < jn
    // element offset of row j at the lane's cells; lanes right of the frame read on into the next row
    uint32_t off = (uint32_t)((ja + STREAM_TOP) * px + STREAM_LEFT + i);
    const uint32_t ring = saddr(ru);
    // stage iteration j (offset o): u, c, d of row j, v of row j - 1
    auto stage = [&](uint32_t o, int slot, uint32_t c) {
        cp16(ring + 4u * slot, u0 + o);
        cp16(ring + 4u * (V + slot), v0 + o);
        cp16(c, a.coef + o);
        cp_async_commit();
    };
    // places in the rings, as floats from ru: the slices' group of three rows now read and the one being
    // filled; the coefficient's group now read, the last, the one before and the one being filled
    int ub0 = 0, ub1 = 3 * FW, cb0 = C, cb1 = C + 3 * FW, cb2 = C + 6 * FW, cbn = C + 9 * FW;
#pragma unroll
    for (int t = 0; t < 6; ++t) stage(off + t * px, t * FW, ring + 4u * ((t < 3 ? cb0 : cbn - 3 * FW) + t * FW));
    // the group's emitters on the rows and columns the warp computes, one to a lane: iteration and column.  More
    // than 32: looked up row by row.  (Always looking them up: 113 us
    // per launch, now 65, against 51 without sources; 32 groups of 512 x 512, history kept.)
    int nem = 0, erow = -1, ecol = 0;
    unsigned eact = 0u;                                    // bit s: row j - s has emitters
    if constexpr (SRC) {
        for (int e0 = 0; e0 < g.gs; e0 += 32) {
            const int q = e0 + lane < g.gs ? em[e0 + lane] : -1, r = q / g.nx - ja, c = q % g.nx - x0;
            const unsigned b = __ballot_sync(FULL, q >= 0 && r >= 0 && r < jn && c >= 0 && c < FW);
            for (unsigned k = b; k; k &= k - 1, ++nem) {   // the nem-th lane takes it
                const int from = __ffs(k) - 1, rk = __shfl_sync(FULL, r, from), ck = __shfl_sync(FULL, c, from);
                if (lane == nem) {
                    erow = rk;
                    ecol = ck;
                }
            }
        }
    }
    const int nrec = gout ? list_receivers(a.rec, ny, y0, yend, x0, max(x0 + FH, 0), min(x0 + FH + FOWN, g.nx), g.nx, rows, ent, lane) : 0;
    // sponge factor: the smaller of the row's and the column's (the damp table grows inwards)
    const float2 dc0 = make_float2(damp_col(g, i), damp_col(g, i + 1)), dc1 = make_float2(damp_col(g, i + 2), damp_col(g, i + 3));
    for (int t = lane; t < jn + 3; t += 32) drow[t] = damp_row(g, ja + t);
    const bool damped = ja < g.sponge_w || yend + T >= ny - g.sponge_w;
    __syncwarp();
    // rolling rows of the levels 0 .. T-1, two pairs a row
    float2 w0[T][2], w1[T][2], w2[T][2];
    const float2 zero = make_float2(0.f, 0.f);
#pragma unroll
    for (int s = 0; s < T; ++s)
#pragma unroll
        for (int v = 0; v < 2; ++v) w0[s][v] = w1[s][v] = w2[s][v] = zero;
    unsigned act = 0u;                                     // bit s: row j - s has receivers
    // one iteration; n: newest rows (written), m, o: the two before; U: position in the group of three
    auto iter = [&](float2 (&n)[T][2], float2 (&m)[T][2], float2 (&o)[T][2], int t, auto uc) {
        constexpr int U = decltype(uc)::value;
        cp_async_wait<FD - 1>();
        const float4 uu = *reinterpret_cast<const float4*>(ru + ub0 + U * FW);
        const float4 vv = *reinterpret_cast<const float4*>(ru + V + ub0 + U * FW);
        n[0][0] = make_float2(uu.x, uu.y);
        n[0][1] = make_float2(uu.z, uu.w);
        if constexpr (SRC) eact = (eact << 1) | (nem > 32 || __any_sync(FULL, erow == t) ? 1u : 0u);
        if (nrec > 0) act = (act << 1) | (t >= T && t < jn - T && rows[t - T].count > 0 ? 1u : 0u);
#pragma unroll
        for (int s = 1; s <= T; ++s) {
            // coefficient of the level's row j - s: staged s iterations before row j's
            const float* cp = ru + (U >= s ? cb0 + (U - s) * FW : U + 3 >= s ? cb1 + (U + 3 - s) * FW : cb2 + (U + 6 - s) * FW);
            const float4 c4 = *reinterpret_cast<const float4*>(cp);
            float2 d0 = dc0, d1 = dc1;
            if (damped) {
                const float dr = drow[t - s < 0 ? 0 : t - s];
                d0 = make_float2(fminf(dc0.x, dr), fminf(dc0.y, dr));
                d1 = make_float2(fminf(dc1.x, dr), fminf(dc1.y, dr));
            }
            const float wl = __shfl_up_sync(FULL, m[s - 1][1].y, 1), er = __shfl_down_sync(FULL, m[s - 1][0].x, 1);
            // level s - 1 at rows j - s + 1 (n), j - s (m), j - s - 1 (o); level s - 2 at row j - s
            const float2 p0 = s == 1 ? make_float2(vv.x, vv.y) : o[s - 2 < 0 ? 0 : s - 2][0];
            const float2 p1 = s == 1 ? make_float2(vv.z, vv.w) : o[s - 2 < 0 ? 0 : s - 2][1];
            const float2 l0 = lap_row(wl, m[s - 1][0], m[s - 1][1].x, o[s - 1][0], n[s - 1][0]);
            const float2 l1 = lap_row(m[s - 1][0].y, m[s - 1][1], er, o[s - 1][1], n[s - 1][1]);
            float2 a0 = pk_fma(make_float2(c4.x, c4.y), l0, twice_less(m[s - 1][0], p0));
            float2 a1 = pk_fma(make_float2(c4.z, c4.w), l1, twice_less(m[s - 1][1], p1));
            if constexpr (SRC) {
                float4 am = make_float4(0.f, 0.f, 0.f, 0.f);
                if ((eact & (1u << s)) && src[s - 1] != 0.f) {
                    auto put = [&](int q) {                // an emitter at column q from the lane's first
                        if (q == 0) am.x = src[s - 1];
                        if (q == 1) am.y = src[s - 1];
                        if (q == 2) am.z = src[s - 1];
                        if (q == 3) am.w = src[s - 1];
                    };
                    if (nem <= 32) {
                        for (unsigned b = __ballot_sync(FULL, erow == t - s); b; b &= b - 1) put(__shfl_sync(FULL, ecol, __ffs(b) - 1) - 4 * lane);
                    } else {
                        const int r = ja + t - s;
                        for (int e = 0; e < g.gs; ++e) put(em[e] / g.nx == r ? em[e] - r * g.nx - i : -1);
                    }
                }
                a0 = pk_fma(d0, a0, make_float2(am.x, am.y));
                a1 = pk_fma(d1, a1, make_float2(am.z, am.w));
            } else {
                a0 = pk_mul(d0, a0);
                a1 = pk_mul(d1, a1);
            }
            if (s < T) {
                n[s < T ? s : 0][0] = a0;
                n[s < T ? s : 0][1] = a1;
            }
            // owned rows: y0 <= j - s < yend
            if (own && (unsigned)(t - T - s) < (unsigned)(jn - 2 * T)) {
                const uint32_t at = off - (uint32_t)(s * px);
                if (hist) __stcs(reinterpret_cast<float4*>(hist + (s - 1) * a.ns + at), make_float4(l0.x, l0.y, l1.x, l1.y));
                if (s == T) *reinterpret_cast<float4*>(o1 + at) = make_float4(a0.x, a0.y, a1.x, a1.y);
                if (T > 1 && s == T - 1) *reinterpret_cast<float4*>(o0 + at) = make_float4(a0.x, a0.y, a1.x, a1.y);
            }
            if (act & (1u << s)) {
                const int r = ja + t - s;
                const RowRec rr = rows[r - y0];
                for (int k = 0; k < rr.count; ++k) {
                    int c;                                 // column and channel
                    if (rr.first + rr.count <= NREC) c = ent[rr.first + k];
                    else {
                        int e = a.rec.rowstart[r];
                        while (a.rec.rcell[e] - r * g.nx < x0 + FH) ++e;
                        e += k;
                        c = (a.rec.rcell[e] - r * g.nx - x0) | a.rec.rchan[e] << 8;
                    }
                    const int q = (c & 255) - 4 * lane;
                    if (q >= 0 && q < 4)
                        gout[(int64_t)s * g.nch + (c >> 8)] = q == 0 ? a0.x : q == 1 ? a0.y : q == 2 ? a1.x : a1.y;
                }
            }
        }
        // the slots just read take iteration j + FD
        stage(off + (uint32_t)FD * px, ub0 + U * FW, ring + 4u * (cb2 + U * FW));
        off += px;
    };
    using U0 = std::integral_constant<int, 0>;
    using U1 = std::integral_constant<int, 1>;
    using U2 = std::integral_constant<int, 2>;
#pragma unroll 1
    for (int t = 0; t < jn; t += 3) {
        iter(w0, w2, w1, t, U0{});
        iter(w1, w0, w2, t + 1, U1{});
        iter(w2, w1, w0, t + 2, U2{});
        const int x = cb2, y = ub0;
        cb2 = cb1;
        cb1 = cb0;
        cb0 = cbn;
        cbn = x;
        ub0 = ub1;
        ub1 = y;
    }
    cp_async_wait<0>();
}

// ---------------------------------------------------------------------------------------------
// Adjoint: z(kz0) .. z(kz0-T+1) with the residual injection and the correlation.
template <int T>
__global__ void __launch_bounds__(SW * 32, 4) k_stream_adj(DevGeo g, StreamAdj a) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, w = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);
    const int ny = g.ny, px = a.px;
    const int id = blockIdx.x * SW + w, strip = id % a.strips, gl = id / a.bands / a.strips;
    const int x0 = strip * AOWN - AH, i = x0 + 2 * lane;
    const int y0 = id / a.strips % a.bands * a.R, yend = min(y0 + a.R, ny);
    // per warp: z1, z2, correlation, L_1 .. L_T [AD][AW]; c, d [AC][AW]; receivers and their residuals
    constexpr int WF = (AD * (3 + T) + 2 * AC) * AW;
    float* const base = reinterpret_cast<float*>(smem4) + w * (WF + MAXR + 16 + NREC + T * NREC);
    float* const rz = base + 2 * lane;                     // this lane's places
    constexpr int Y = 3 * AW, KK = 6 * AW, LL = 9 * AW, C = (9 + 3 * T) * AW, DD = AC * AW;
    RowRec* const rows = reinterpret_cast<RowRec*>(base + WF);
    int* const ent = reinterpret_cast<int*>(base + WF + MAXR + 16);
    float* const val = base + WF + MAXR + 16 + NREC;   // [T][NREC]
    if (gl >= a.ng) return;
    const bool own = i >= 0 && i < g.nx && lane >= 2 && lane <= 29;
    const float* const z1 = a.in1 + gl * a.instride;
    const float* const z2 = a.in0 + gl * a.instride - px;  // row j - 1 at row j's offset
    float* const o1 = a.out1 + gl * a.instride;
    float* const o0 = T > 1 ? a.out0 + gl * a.instride : nullptr;
    float* const corr = a.corr + gl * a.cstride;
    const float* const rr = a.rr + gl * a.rrstride + (int64_t)a.kz0 * g.nch;
    const float* const hist = a.hist + gl * a.hstride + (int64_t)(a.kz0 - 1 - a.qlo) * a.ns;   // L of level 1
    const int yr = y0 - T, jn = yend - y0 + 2 * T;         // iterations j = yr + t, t < jn
    uint32_t off = (uint32_t)((yr + STREAM_TOP) * px + STREAM_LEFT + i);
    // Copies are of 16 bytes, half a warp to a row: lanes 0-15 bring the first and lanes 16-31 the second
    // of (z1, c), (z2, d), (correlation, L_1), (L_2, L_3), (L_4, -); z2, the correlation and L_s are of
    // the rows j - 1 and j - s, c and d of row j like z1.  (Copies of 8 bytes, a lane its own cells, take
    // twice the instructions and pass through L1.)
    const int half = lane >> 4, ch = 4 * (lane & 15);
    const uint32_t shift = (uint32_t)(x0 + ch - i);        // from the lane's cells to its chunk's
    const float* const s0 = half ? a.coef : z1;
    const float* const s1 = half ? a.dmap : z2;
    const float* const s2 = half ? hist - px : corr - px;
    const float* const s3 = half ? hist - 2 * a.ns - 3 * px : hist - a.ns - 2 * px;
    const float* const s4 = hist - 3 * a.ns - 4 * px;
    const uint32_t ring = saddr(base) + 4u * ch;
    auto stage = [&](uint32_t o, int slot, int c) {        // c: the coefficient's place, as floats from base
        o += shift;
        cp16(ring + 4u * (half ? c : slot * AW), s0 + o);
        cp16(ring + 4u * (half ? c + DD : Y + slot * AW), s1 + o);
        cp16(ring + 4u * ((half ? LL : KK) + slot * AW), s2 + o);
        if (T == 4) {
            cp16(ring + 4u * (LL + (half ? 6 : 3) * AW + slot * AW), s3 + o);
            if (!half) cp16(ring + 4u * (LL + 9 * AW + slot * AW), s4 + o);
        } else if (T == 2) {
            if (!half) cp16(ring + 4u * (LL + 3 * AW + slot * AW), s3 + o);
        }
        cp_async_commit();
    };
    int cb0 = C, cb1 = C + 3 * AW, cb2 = C + 6 * AW;
#pragma unroll
    for (int t = 0; t < 3; ++t) stage(off + t * px, t, cb0 + t * AW);
    const float2 zero = make_float2(0.f, 0.f);
    float2 zn[T], zm[T], zo[T], pn[T], pm[T], po[T], cr[T + 1];
#pragma unroll
    for (int s = 0; s < T; ++s) zn[s] = zm[s] = zo[s] = pn[s] = pm[s] = po[s] = zero;
#pragma unroll
    for (int s = 0; s <= T; ++s) cr[s] = zero;
    unsigned act = 0u;
    // receivers of every cell the warp computes (halo included), rows y0 - T .. yend + T - 1
    const int nrec = list_receivers(a.rec, ny, yr, yend + T, x0, max(x0, 0), min(x0 + AW, g.nx), g.nx, rows, ent, lane);
    const int keep = min(nrec, NREC);
    for (int e = lane; e < keep; e += 32)
#pragma unroll
        for (int s = 0; s < T; ++s) cp4(val + s * NREC + e, rr - (int64_t)s * g.nch + (ent[e] >> 8));
    cp_async_commit();
    cp_async_wait<0>();                                    // the residuals, and the first rows
    __syncwarp();
    auto iter = [&](float2 (&Zn)[T], float2 (&Zm)[T], float2 (&Zo)[T], float2 (&Pn)[T], float2 (&Pm)[T], float2 (&Po)[T], int t,
                    auto uc) {
        constexpr int U = decltype(uc)::value;
        cp_async_wait<2>();
        __syncwarp();                                      // every lane's copies of row j are there
        Zn[0] = *reinterpret_cast<const float2*>(rz + U * AW);
        Pn[0] = pk_mul(*reinterpret_cast<const float2*>(rz + cb0 + U * AW), Zn[0]);
        if (nrec > 0) act = (act << 1) | (t < jn && rows[t].count > 0 ? 1u : 0u);
        float2 zs[T + 1];
#pragma unroll
        for (int s = 1; s <= T; ++s) {
            const float* cp = rz + (U >= s ? cb0 + (U - s) * AW : U + 3 >= s ? cb1 + (U + 3 - s) * AW : cb2 + (U + 6 - s) * AW);
            const float2 d = *reinterpret_cast<const float2*>(cp + DD);
            const float pw = __shfl_up_sync(FULL, Pm[s - 1].y, 1), pe = __shfl_down_sync(FULL, Pm[s - 1].x, 1);
            const float2 zz = s == 1 ? *reinterpret_cast<const float2*>(rz + Y + U * AW) : Zo[s - 2 < 0 ? 0 : s - 2];
            float2 x = pk_add(twice_less(Zm[s - 1], zz), lap_row(pw, Pm[s - 1], pe, Po[s - 1], Pn[s - 1]));
            if (act & (1u << s)) {                         // residuals of the row's receivers
                const int r = yr + t - s;
                const RowRec q = rows[t - s];
                for (int k = 0; k < q.count; ++k) {
                    int c;
                    float v;
                    if (q.first + q.count <= NREC) {
                        c = (ent[q.first + k] & 255) - 2 * lane;
                        v = val[(s - 1) * NREC + q.first + k];
                    } else {
                        int e = a.rec.rowstart[r];
                        while (a.rec.rcell[e] - r * g.nx < x0) ++e;
                        e += k;
                        c = a.rec.rcell[e] - r * g.nx - i;
                        v = rr[a.rec.rchan[e] - (int64_t)(s - 1) * g.nch];
                    }
                    if (c == 0) x.x = __fadd_rn(x.x, v);
                    if (c == 1) x.y = __fadd_rn(x.y, v);
                }
            }
            zs[s] = pk_mul(d, x);
            if (s < T) {
                Zn[s < T ? s : 0] = zs[s];
                Pn[s < T ? s : 0] = pk_mul(*reinterpret_cast<const float2*>(cp), zs[s]);
            }
            if (s >= T - 1 && s >= 1 && own && (unsigned)(t - T - s) < (unsigned)(jn - 2 * T)) {
                const uint32_t at = off - (uint32_t)(s * px);
                if (s == T) *reinterpret_cast<float2*>(o1 + at) = zs[s];
                if (T > 1 && s == T - 1) *reinterpret_cast<float2*>(o0 + at) = zs[s];
            }
        }
        // the correlation of row j - s after level s: that of the same row after level s - 1, one
        // iteration ago
        cr[0] = *reinterpret_cast<const float2*>(rz + KK + U * AW);
#pragma unroll
        for (int s = T; s >= 1; --s) {
            const float2 c0 = s == 1 ? cr[0] : cr[s - 1];
            cr[s] = pk_fma(zs[s], *reinterpret_cast<const float2*>(rz + LL + ((s - 1) * 3 + U) * AW), c0);
        }
        if (own && (unsigned)(t - 2 * T) < (unsigned)(jn - 2 * T))
            *reinterpret_cast<float2*>(corr + (off - (uint32_t)(T * px))) = cr[T];
        __syncwarp();                                      // the slots have been read
        stage(off + 3u * px, U, cb2 + U * AW);
        off += px;
    };
    using U0 = std::integral_constant<int, 0>;
    using U1 = std::integral_constant<int, 1>;
    using U2 = std::integral_constant<int, 2>;
#pragma unroll 1
    for (int t = 0; t < jn; t += 3) {
        iter(zn, zo, zm, pn, po, pm, t, U0{});
        iter(zm, zn, zo, pm, pn, po, t + 1, U1{});
        iter(zo, zm, zn, po, pm, pn, t + 2, U2{});
        const int x = cb2;
        cb2 = cb1;
        cb1 = cb0;
        cb0 = x;
    }
    cp_async_wait<0>();
}

// Simulated samples in rr -> residuals meas - sample (with the record noise), and the sum of their
// squares per (group, step) in the order of k_resid_parts.
__global__ void __launch_bounds__(256) k_resid_meas(DevGeo g, float* __restrict__ rr, const float* __restrict__ meas, int g0,
                                                   int64_t rows, double* part) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int k = (int)(row % g.nt), gl = (int)(row / g.nt);
    const bool noisy = g.noise_key;
    const uint64_t key = noisy ? *g.noise_key : 0;
    float* r = rr + row * g.nch;
    const float* m = meas + row * g.nch;
    double v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        v[j] = 0.0;
        for (int c = lane + 32 * j; c < g.nch; c += 256) {
            float e = 0.f;
            if (k >= 2) {
                float x = r[c];
                if (noisy) x = __fmul_rn(x, noise_factor(key, g.noise_level, g0 + gl, k, c));   // not contracted
                e = m[c] - x;
            }
            r[c] = e;
            v[j] += (double)e * (double)e;
        }
    }
#pragma unroll
    for (int w = 4; w > 0; w >>= 1)
#pragma unroll
        for (int j = 0; j < w; ++j) v[j] += v[j + w];
    for (int w = 16; w > 0; w >>= 1) v[0] += __shfl_down_sync(FULL, v[0], w);
    if (lane == 0) part[row] = v[0];
}

// Natural planes of nx x ny cells into the frame of guard cells (zeroed here) and back.
__global__ void k_frame(float* __restrict__ dst, const float* __restrict__ src, int nx, int ny, int px, int64_t ns) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < ns; q += (int64_t)gridDim.x * blockDim.x) {
        const int y = (int)(q / px) - STREAM_TOP, x = (int)(q % px) - STREAM_LEFT;
        dst[q] = x >= 0 && x < nx && y >= 0 && y < ny ? src[(int64_t)y * nx + x] : 0.f;
    }
}
__global__ void k_unframe(float* __restrict__ dst, int64_t dstride, const float* __restrict__ src, int64_t sstride, int nx, int ny,
                          int px) {
    float* d = dst + blockIdx.y * dstride;
    const float* s = src + blockIdx.y * sstride + (int64_t)STREAM_TOP * px + STREAM_LEFT;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < (int64_t)nx * ny; q += (int64_t)gridDim.x * blockDim.x)
        d[q] = s[q / nx * px + q % nx];
}
// Zeroes the guard cells of planes (one per blockIdx.y, ns floats apart): the kernels of other passes
// use the same buffers without a frame.  The guard cells are the head of the plane, the gaps between the
// rows (one row's right guard and the next one's left) and the tail; only they are touched.
__global__ void k_zero_frame(float* __restrict__ p, int nx, int ny, int px, int64_t ns) {
    float* d = p + blockIdx.y * ns;
    const int head = STREAM_TOP * px + STREAM_LEFT, gap = px - nx, t = blockIdx.x * blockDim.x + threadIdx.x,
              n = gridDim.x * blockDim.x;
    for (int q = t; q < head; q += n) d[q] = 0.f;
    for (int64_t q = t; q < (int64_t)(ny - 1) * gap; q += n) d[head + q / gap * px + nx + q % gap] = 0.f;
    for (int64_t q = head + (int64_t)(ny - 1) * px + nx + t; q < ns; q += n) d[q] = 0.f;
}

// Four blocks fit an SM's 228 KB with 1 KB each for the system (with three the gradient share of 8 groups of 2048 x
// 2048 took 59.5 ms, not 56).
constexpr size_t fwd_smem() { return 4 * (size_t)SW * ((2 * FD + FC) * FW + 2 * MAXR + 16 + NREC); }
constexpr size_t adj_smem(int T) { return 4 * (size_t)SW * ((AD * (3 + T) + 2 * AC) * AW + MAXR + 16 + NREC + T * NREC); }
static_assert(4 * (fwd_smem() + 1024) <= 228 * 1024 && 4 * (adj_smem(4) + 1024) <= 228 * 1024, "four blocks per SM");

// Rows of a band (152: the SMs of a GB300).  A block's time grows with the R + 2 T rows it computes; four blocks are resident on an
// SM, and an SM with fewer than about 2.5 waits on latency, so a last wave of one block per SM costs as much
// as one of 2.5.  Measured forward us per step (without history), 32 groups of 512 x 512: R 28, 36, 64, 76,
// 104: 11.0, 8.9, 11.4, 11.4, 15.4; 8 groups of 2048 x 2048: 29.4, 28.7, 27.2, 28.0, 32.8.  Adjoint: 24.7,
// 24.0, 24.6, 23.0, 21.7 and 86, 83, 78, 74, 76.
int band_rows(int ny, int strips, int ng, int T) {
    int best = 16;
    double least = 1e300;
    for (int R = 8; R <= MAXR - 8; ++R) {
        const double blocks = std::ceil((double)strips * ng * ((ny + R - 1) / R) / SW);
        const double per_sm = std::ceil(blocks / 152.0), waves = std::floor(per_sm / 4.0), tail = per_sm - 4.0 * waves;
        const double t = (4.0 * waves + (tail > 0.0 ? std::max(2.5, tail) : 0.0)) * (std::min(R, ny) + 2 * T);
        if (t < least) {
            least = t;
            best = R;
        }
    }
    return best;
}

template <typename Args>
int cut(const DevGeo& g, Args& a, int owned) {   // blocks of the launch
    a.strips = (g.nx + owned - 1) / owned;
    a.R = band_rows(g.ny, a.strips, a.ng, a.T);
    a.bands = (g.ny + a.R - 1) / a.R;
    return (int)(((int64_t)a.strips * a.bands * a.ng + SW - 1) / SW);
}
template <int T, bool SRC>
void go_fwd(const DevGeo& g, StreamFwd a, void* st) {
    const int blocks = cut(g, a, FOWN);
    cudaFuncSetAttribute(k_stream_fwd<T, SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem());
    k_stream_fwd<T, SRC><<<blocks, SW * 32, fwd_smem(), (cudaStream_t)st>>>(g, a);
}
template <int T>
void go_adj(const DevGeo& g, StreamAdj a, void* st) {
    const int blocks = cut(g, a, AOWN);
    cudaFuncSetAttribute(k_stream_adj<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)adj_smem(T));
    k_stream_adj<T><<<blocks, SW * 32, adj_smem(T), (cudaStream_t)st>>>(g, a);
}
}  // namespace

int stream_pitch(int nx) { return ((nx + 7) & ~7) + 2 * STREAM_LEFT; }
int64_t stream_slice(int nx, int ny) {
    // 128: lanes to the right of the last strip read that far past the last guard row
    return (int64_t)stream_pitch(nx) * (ny + STREAM_TOP + STREAM_BOTTOM) + 128;
}

void launch_stream_fwd(const DevGeo& g, const StreamFwd& a, void* st) {
    const bool src = a.k0 < g.n_src_steps;
    if (a.T == 4) src ? go_fwd<4, true>(g, a, st) : go_fwd<4, false>(g, a, st);
    else if (a.T == 2) src ? go_fwd<2, true>(g, a, st) : go_fwd<2, false>(g, a, st);
    else src ? go_fwd<1, true>(g, a, st) : go_fwd<1, false>(g, a, st);
}
int64_t launch_stream_steps(const DevGeo& g, StreamFwd a, StreamState& st, int T, float* ring, int64_t rstride, float* end0,
                            float* end1, int64_t endstride, void* stream) {
    int64_t n = 0;
    for (; T > 0; T -= a.T, ++n) {
        // the last launch advances two or more steps where there are any, so both slices of the end state come
        // from one launch
        a.T = T >= 6 || T == 4 ? 4 : T % 2 ? 1 : 2;
        a.in0 = st.p0;
        a.in1 = st.p1;
        a.in0stride = st.s0;
        a.in1stride = st.s1;
        if (T == a.T && end0) {
            a.out0 = end0;
            a.out1 = end1;
            a.outstride = endstride;
        } else {   // two ring slots the inputs are not in
            float* free[2] = {nullptr, nullptr};
            for (int k = 0, f = 0; k < STREAM_RING && f < 2; ++k) {
                float* s = ring + k * a.ns;
                if (s != st.p0 && s != st.p1) free[f++] = s;
            }
            a.out0 = free[0];
            a.out1 = free[1];
            a.outstride = rstride;
        }
        launch_stream_fwd(g, a, stream);
        if (a.T == 1) st = StreamState{st.p1, a.out1, st.s1, a.outstride};
        else st = StreamState{a.out0, a.out1, a.outstride, a.outstride};
        a.k0 += a.T;
    }
    return n;
}
void launch_stream_adj(const DevGeo& g, const StreamAdj& a, void* st) {
    if (a.T == 4) go_adj<4>(g, a, st);
    else if (a.T == 2) go_adj<2>(g, a, st);
    else go_adj<1>(g, a, st);
}
void launch_resid_meas(const DevGeo& g, float* rr, const float* meas, int g0, int ng, double* part, void* stream) {
    const int64_t rows = (int64_t)ng * g.nt;
    k_resid_meas<<<(unsigned)((rows + 7) / 8), 256, 0, (cudaStream_t)stream>>>(g, rr, meas, g0, rows, part);
}
void launch_frame(float* dst, const float* src, int nx, int ny, void* stream) {
    k_frame<<<608, 256, 0, (cudaStream_t)stream>>>(dst, src, nx, ny, stream_pitch(nx), stream_slice(nx, ny));
}
void launch_unframe(float* dst, int64_t dstride, const float* src, int64_t sstride, int nx, int ny, int planes, void* stream) {
    k_unframe<<<dim3(152, planes), 256, 0, (cudaStream_t)stream>>>(dst, dstride, src, sstride, nx, ny, stream_pitch(nx));
}
void launch_zero_frame(float* p, int64_t planes, int nx, int ny, void* stream) {
    for (int64_t k = 0; k < planes; k += 32768)
        k_zero_frame<<<dim3(4, (unsigned)std::min<int64_t>(32768, planes - k)), 256, 0, (cudaStream_t)stream>>>(
            p + k * stream_slice(nx, ny), nx, ny, stream_pitch(nx), stream_slice(nx, ny));
}

}  // namespace tomo
