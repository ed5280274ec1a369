// resident_ref.cuh -- cluster-resident sweeps of the reference profile.
//
// The organisation of resident.cuh; what differs is the arithmetic (the reference's
// operation order, every operation rounded, as kernels.cu) and the edges: one-way absorbing edges
// in the forward sweep, edge copies and sensor lines in the adjoint.  A row's edge or sensor value
// depends on the row beside it, so the rows are dealt out in pairs: (0, 1), (lo, lo+1), (hi-1, hi)
// and (ny-2, ny-1) each share a warp, and a warp may hold a single row where the rows between
// two such pairs are odd in number (ref_warps).  A single row's second slot mirrors the row above
// it, so the first slot's arithmetic is the same in every warp.
//
// Edge columns are evaluated by the two lanes that own them, from the rows the warp published
// (the slices u(m-1) and u(m-2) of its own rows are both still in shared memory), and put into
// place; the cell beyond the right edge keeps a copy of the edge, which is the neighbour the
// clamped Laplacian reads.
//
// Measured (one GB300): the 192 x 192 problem of 401 steps, 64 groups: 5.7 / 6.4 us per forward /
// adjoint step (per-cell kernels: 13 us with the gather, 22), an iteration 5.6 ms (14.0); one group
// of it on a cluster of 14 blocks 0.93 / 1.07 us (9.3 us for the three launches of a step before),
// a sequential iteration of 32 groups 27.0 ms (119.6); data generation 2.2 ms (5.2).  What bounds a
// step: the instruction stream of a warp's two rows.  ncu, one group of 192 x 192 on 14 blocks of 7 warps:
// 327 instructions per warp and step forward, 421 adjoint, at 1.75 warps per scheduler; 29 and 33 % of the cycles
// issue, fixed latencies (1.2 and 1.5 cycles per issue) and forward the block barrier (1.1) the largest stalls.
#pragma once
#include "resident.cuh"

namespace tomo {
namespace {

__device__ __forceinline__ float xm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float xa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float xs(float a, float b) { return __fsub_rn(a, b); }

// Coefficients of the one-way edge update at a cell of Courant number r (sirt-mimo.cu:565-587).
struct RefEdge {
    float k1, k2, k3, k4, k5;
    __device__ __forceinline__ void set(float r) {
        const float r2 = xm(r, r), tr = xm(2.f, r);
        k1 = xs(xs(2.f, tr), r2);
        k2 = xm(tr, xa(1.f, r));
        k3 = r2;
        k4 = xs(tr, 1.f);
        k5 = tr;
    }
    // u, ua, ub: the cell and the two inside it at k; up, upa: at k - 1
    __device__ __forceinline__ float operator()(float u, float ua, float ub, float up, float upa) const {
        return xs(xa(xs(xa(xm(k1, u), xm(k2, ua)), xm(k3, ub)), xm(k4, up)), xm(k5, upa));
    }
};

// Rows of a warp: first row and how many (1 or 2; 0 for a warp past the last).
struct RefRows {
    int j0, n;
};
__device__ __forceinline__ RefRows ref_rows(const int32_t* table, int nwarps, int gw) {
    if (gw >= nwarps) return RefRows{1 << 20, 0};
    const int v = table[gw];
    return RefRows{v & 0xffff, v >> 16};
}

template <int CPL>
__device__ __forceinline__ void put_cell(float2 (&x)[CPL / 2], int i, float v) {
#pragma unroll
    for (int k = 0; k < CPL / 2; ++k) {
        if (i == 2 * k) x[k].x = v;
        if (i == 2 * k + 1) x[k].y = v;
    }
}
// Cell i (the same in every lane) and the one after it, in the lanes with `on`.
template <int CPL>
__device__ __forceinline__ void put_edge(float2 (&x)[CPL / 2], int i, bool on, float v) {
#pragma unroll
    for (int k = 0; k < CPL; ++k)
        if (i == k) {
            float& o = k % 2 == 0 ? x[k / 2].x : x[k / 2].y;
            o = on ? v : o;
            if (k + 1 < CPL) {
                float& p = k % 2 == 0 ? x[k / 2].y : x[(k / 2 + 1) % (CPL / 2)].x;
                p = on ? v : p;
            }
        }
}
template <int CPL>
__device__ __forceinline__ float get_cell(const float2 (&x)[CPL / 2], int i) {
    float v = x[0].x;
#pragma unroll
    for (int k = 0; k < CPL / 2; ++k) {
        if (i == 2 * k) v = x[k].x;
        if (i == 2 * k + 1) v = x[k].y;
    }
    return v;
}

// Corners of an edge row ex (its Laplacian lx, the inner row's lin): the mean of the two edge
// neighbours, side being the one in the inner row.  lr, ie: lane and cell of the right edge.
template <int CPL>
__device__ __forceinline__ void ref_corners(float2 (&ex)[CPL / 2], float2 (&lx)[CPL / 2], const float2 (&lin)[CPL / 2],
                                            float side, int lane, int lr, int ie) {
    const float in_up = __shfl_up_sync(FULL, ex[CPL / 2 - 1].y, 1), lin_up = __shfl_up_sync(FULL, lx[CPL / 2 - 1].y, 1);
    if (lane == 0) {
        ex[0].x = xm(0.5f, xa(side, ex[0].y));
        lx[0].x = xm(0.5f, xa(lin[0].x, lx[0].y));
    }
    if (lane == lr) {
        const float c = xm(0.5f, xa(side, ie > 0 ? get_cell<CPL>(ex, ie - 1) : in_up));
        put_cell<CPL>(ex, ie, c);
        put_cell<CPL>(ex, ie + 1, c);
        put_cell<CPL>(lx, ie, xm(0.5f, xa(get_cell<CPL>(lin, ie), ie > 0 ? get_cell<CPL>(lx, ie - 1) : lin_up)));
    }
    __syncwarp();
}

template <int CPL, int RPW, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_ref_fwd(DevGeo g, ResFwd a) {
    using F = Frag<CPL>;
    constexpr int NP = F::NP, ROW = F::ROW;
    static_assert(RPW == 2, "rows come in pairs");
    extern __shared__ __align__(1024) unsigned char smraw[];
    const int W = blockDim.x >> 5, lane = threadIdx.x & 31, w = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);
    const ResSmem sm = res_smem<CPL, RPW, true>(smraw, W);
    const int rank = (int)cluster_rank(), cs = a.cs, gl = blockIdx.x / cs;
    const int nx = g.nx, ny = g.ny, ggl = a.g0 + gl, T = a.T;
    const RefRows me = ref_rows(a.warps, a.nwarps, rank * W + w);
    const int j0 = me.j0;
    const bool single = me.n == 1, first_row = j0 == 0, last_row = j0 == ny - 2;
    res_setup(sm, rank, cs, 4 * ROW, 4u * ROW, a.w.extra_tx);
    ResLinks<CPL> lk;
    lk.init(sm, rank, cs, w == 0, w == W - 1, a.w.wait_ns);
    lk.single = single;
    const int64_t fbase = (int64_t)j0 * ROW;
    const int xr = nx - 1, lr = xr / CPL, ie = xr - lr * CPL;       // right edge: column, lane, cell of the lane
    const bool edge = lane == 0 || lane == lr;
    float2 cc[RPW][NP], ua[RPW][NP], ub[RPW][NP];
    RefEdge ke[RPW];           // edge columns (lanes 0 and lr)
    auto courant = [&](int j, int x) { return __fdiv_rn(xm(a.rcoef[(int64_t)j * nx + x], kRefDT), kRefH); };
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int j = j0 + r;
        const bool in = r < me.n;
        F::load_nat(cc[r], a.coef + (int64_t)j * nx, lane, nx, in);
#pragma unroll
        for (int v = 0; v < NP; ++v) ua[r][v] = ub[r][v] = make_float2(0.f, 0.f);   // u(k0), u(k0-1)
        if (a.in0 && in) {
            F::load(ub[r], a.in0 + gl * a.instride + (int64_t)j * ROW, lane);
            F::load(ua[r], a.in1 + gl * a.instride + (int64_t)j * ROW, lane);
        }
        ke[r].set(in && edge ? courant(j, lane == 0 ? 0 : xr) : 0.f);
    }
    // the edge rows' Courant numbers (rows 0 and ny - 1), and the emission box of the group
    float* const erow = sm.val + (last_row ? ROW : 0);
    if (first_row || last_row)
        for (int v = 0; v < CPL; ++v) {
            const int x = CPL * lane + v;
            erow[F::at(lane, v / 2) + v % 2] = x < nx ? courant(last_row ? ny - 1 : 0, x) : 0.f;
        }
    const int32_t* const box = g.box + 4 * ggl;
    // receivers of the block (consecutive in row order)
    const RefRows blo = ref_rows(a.warps, a.nwarps, rank * W), bhi = ref_rows(a.warps, a.nwarps, min(rank * W + W, a.nwarps) - 1);
    const int n0 = a.gout ? a.rowstart[blo.j0] : 0, n1 = a.gout ? a.rowstart[bhi.j0 + bhi.n] : 0;
    const bool noisy = a.gmeas && g.noise_key;
    const uint64_t key = noisy ? *g.noise_key : 0;
    const int64_t rbase = (int64_t)gl * g.nt * g.nch;
    auto rec_off = [&](int n) {                            // place of receiver n in the published rows, parity 0
        const int q = a.rcell[n], j = q / nx;
        return (a.rowslot[j] - rank * W * RPW) * 2 * ROW + F::col(q - j * nx);
    };
    int roff = 0, rch = 0;
    const int ri = 32 * ((w + W - 1) % W) + lane;
    const bool rec = n0 + ri < n1, rec_more = n0 + (int)blockDim.x < n1;
    if (rec) {
        roff = rec_off(n0 + ri);
        rch = a.rchan[n0 + ri];
    }
    const bool rec_warp = n0 + ri - lane < n1, meas = rec && a.gmeas;
    float* op = rec ? a.gout + rbase + (int64_t)(a.k0 + 1) * g.nch + rch : nullptr;         // slice k0 + 1
    const float* mp = meas ? a.gmeas + rbase + (int64_t)(a.k0 + 1) * g.nch + rch : nullptr;
    const float* const pub0 = sm.xch + roff;
    float* const mring = sm.ring + threadIdx.x;
    int mi = 0, mleft = meas ? T : 0;
    auto request = [&](int i) {
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
                const int ch = a.rchan[n];
                const int64_t o = rbase + (int64_t)m * g.nch + ch;
                put(sm.xch[rec_off(n) + P * ROW], a.gmeas ? a.gmeas[o] : 0.f, a.gout + o, m, ch);
            }
        }
    };
    float* const xw = sm.xch + w * RPW * 2 * ROW;
    auto publish = [&](const float2 (&x)[RPW][NP], auto pc, bool remote) {
        constexpr int P = decltype(pc)::value;
        F::store(xw + P * ROW, x[0], lane);
        if (single) F::store(xw + (2 + P) * ROW, x[0], lane);
        else F::store(xw + (2 + P) * ROW, x[1], lane);
        if (remote) lk.template send<P>(x[0], x[1], lane);
    };
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;
    if (meas)
        for (int i = 0; i < RES_MEAS; ++i) request(i);
    __syncthreads();
    cluster_sync();
    publish(ub, P1{}, false);                              // u(k0-1): only this warp's edge columns read it
    publish(ua, P0{}, true);
    __syncthreads();

    const float* const srow = w > 0 ? xw - 2 * ROW : sm.halo;
    const float* const nrow = w < W - 1 ? xw + RPW * 2 * ROW : sm.halo + 2 * ROW;
    // published places of the edge column and the two columns inside it
    const int eq = F::col(lane == 0 ? 0 : xr), ea = F::col(lane == 0 ? 1 : xr - 1), eb = F::col(lane == 0 ? 2 : xr - 2);
    const int tkeep = a.hist ? a.qlo - a.k0 + 1 : T + 1;
    float* hp = a.hist ? a.hist + gl * a.hstride + fbase : nullptr;
    // one step (see k_res_fwd); em: the source amplitudes v v DT DT of the cells inside the box
    auto step = [&](float2 (&cur)[RPW][NP], float2 (&prv)[RPW][NP], int t, auto pc, auto src_c, float s1, float s2,
                    const float2 (&em)[RPW][NP]) {
        constexpr int P = decltype(pc)::value;
        constexpr bool SRC = decltype(src_c)::value;
        lk.template recv<P>(sm, t, lane);
        float2 sb[NP], nb[NP];
        F::load(sb, srow + P * ROW, lane);
        F::load(nb, nrow + P * ROW, lane);
        if (single) {
#pragma unroll
            for (int v = 0; v < NP; ++v) cur[1][v] = nb[v];
        }
        // edge columns of u(m), from the published slices u(m-1) and u(m-2)
        float ev[2];
        ev[0] = ev[1] = 0.f;
        if (edge) {
#pragma unroll
            for (int r = 0; r < RPW; ++r) {
                const float *c = xw + (2 * r + P) * ROW, *p = xw + (2 * r + (P ^ 1)) * ROW;
                ev[r] = ke[r](c[eq], c[ea], c[eb], p[eq], p[ea]);
            }
        }
        __syncwarp();
        // edge rows: the one-way update along y, before the rows are overwritten
        float2 er0[NP];
        if (first_row || last_row) {
            float2 rc[NP];
            F::load(rc, erow, lane);
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                RefEdge k;
                k.set(rc[v].x);
                er0[v].x = first_row ? k(cur[0][v].x, cur[1][v].x, nb[v].x, prv[0][v].x, prv[1][v].x)
                                     : k(cur[1][v].x, cur[0][v].x, sb[v].x, prv[1][v].x, prv[0][v].x);
                k.set(rc[v].y);
                er0[v].y = first_row ? k(cur[0][v].y, cur[1][v].y, nb[v].y, prv[0][v].y, prv[1][v].y)
                                     : k(cur[1][v].y, cur[0][v].y, sb[v].y, prv[1][v].y, prv[0][v].y);
            }
        }
        const bool keep = t >= tkeep;
        float2 lap[RPW][NP];
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const float wr = __shfl_up_sync(FULL, cur[r][NP - 1].y, 1), er = __shfl_down_sync(FULL, cur[r][0].x, 1);
            // clamped at the edges (the clamped values only reach the history)
            const float wl = lane == 0 ? cur[r][0].x : wr;
            const float el = lane == lr && ie == CPL - 1 ? cur[r][NP - 1].y : er;
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                const float2 u = cur[r][v];
                const float2 s = r == 0 ? (first_row ? u : sb[v]) : cur[0][v];
                const float2 n = r == 1 ? (last_row ? u : nb[v]) : cur[1][v];
                const float we = v > 0 ? cur[r][v - 1].y : wl, ee = v + 1 < NP ? cur[r][v + 1].x : el;
                // r r (((E + W) + S) + N) + (2 - 4 r r) u - up
                const float2 nbs = pk_add(pk_add(make_float2(xa(u.y, we), xa(ee, u.x)), s), n);
                const float2 c = cc[r][v];
                // (scalar products: a packed product that feeds a packed sum is contracted with it)
                float2 x = pk_sub(pk_add(mul2(c, nbs), mul2(pk_fma(make_float2(-4.f, -4.f), c, make_float2(2.f, 2.f)), u)),
                                  prv[r][v]);
                if constexpr (SRC) {
                    const float2 am = em[r][v];
                    if (am.x != 0.f) x.x = xa(x.x, xm(xm(am.x, s1), s2));
                    if (am.y != 0.f) x.y = xa(x.y, xm(xm(am.y, s1), s2));
                }
                // (((S + N) + W) + E) - 4 u
                const float2 sn = pk_add(s, n);
                lap[r][v] = pk_fma(make_float2(-4.f, -4.f), u,
                                   make_float2(xa(xa(sn.x, we), u.y), xa(xa(sn.y, u.x), ee)));
                prv[r][v] = x;
            }
        }
        if (first_row) {
#pragma unroll
            for (int v = 0; v < NP; ++v) prv[0][v] = er0[v];
        }
        if (last_row) {
#pragma unroll
            for (int v = 0; v < NP; ++v) prv[1][v] = er0[v];
        }
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            if (lane == 0) prv[r][0].x = ev[r];
            put_edge<CPL>(prv[r], ie, lane == lr, ev[r]);
        }
        // corners: the mean of the two edge neighbours; and the Laplacian's at the corners of u(m-1)
        if (first_row) ref_corners<CPL>(prv[0], lap[0], lap[1], ev[1], lane, lr, ie);
        if (last_row) ref_corners<CPL>(prv[1], lap[1], lap[0], ev[0], lane, lr, ie);
        publish(prv, std::integral_constant<int, (P ^ 1)>{}, true);
        if (keep) {
#pragma unroll
            for (int r = 0; r < RPW; ++r)
                if (r < me.n) F::store(hp + r * ROW, lap[r], lane);
            hp += a.ns;
        }
    };
    int t = 1;
    bool live = true;
    {
        float2 em[RPW][NP];
#pragma unroll
        for (int r = 0; r < RPW; ++r)
#pragma unroll
            for (int v = 0; v < NP; ++v) em[r][v] = make_float2(0.f, 0.f);
        if (a.k0 < g.n_src_steps) {
            const int i0 = max(box[0], 1), i1 = min(box[1], nx - 2), y0 = max(box[2], 1), y1 = min(box[3], ny - 2);
#pragma unroll
            for (int r = 0; r < RPW; ++r) {
                const int j = j0 + r;
                if (r >= me.n || j < y0 || j > y1) continue;
#pragma unroll
                for (int v = 0; v < CPL; ++v) {
                    const int x = CPL * lane + v;
                    float am = 0.f;
                    if (x >= i0 && x <= i1) {
                        const float vel = a.rcoef[(int64_t)j * nx + x];
                        am = xm(xm(xm(vel, vel), kRefDT), kRefDT);
                    }
                    if (v % 2 == 0) em[r][v / 2].x = am;
                    else em[r][v / 2].y = am;
                }
            }
        }
        const int ns = g.n_src_steps, tsrc = max(1, min(T, ns - a.k0));
#pragma unroll 1
        for (; t <= tsrc && live; t += 2) {
            const int k = a.k0 + t - 1, failed = res_failed(sm, t);
            if (k < ns) step(ua, ub, t, P0{}, std::true_type{}, g.src[k], g.src[ns + k], em);
            else step(ua, ub, t, P0{}, std::false_type{}, 0.f, 0.f, em);
            if (t > 1) record(k, P0{});
            __syncthreads();
            if (t < T) {
                if (k + 1 < ns) step(ub, ua, t + 1, P1{}, std::true_type{}, g.src[k + 1], g.src[ns + k + 1], em);
                else step(ub, ua, t + 1, P1{}, std::false_type{}, 0.f, 0.f, em);
                record(k + 1, P1{});
                __syncthreads();
            }
            live = failed == 0;
            if (a.ckpt && t + 1 <= T) res_checkpoint<CPL, RPW>(a, gl, fbase, t + 1, ub, ua, lane, me.n);
        }
    }
    int tck = a.ckpt ? res_next_checkpoint(a, t) : T + 1;
#pragma unroll 1
    for (; t + 1 <= T && live; t += 2) {
        const int failed = res_failed(sm, t);
        step(ua, ub, t, P0{}, std::false_type{}, 0.f, 0.f, ua);
        record(a.k0 + t - 1, P0{});
        __syncthreads();
        step(ub, ua, t + 1, P1{}, std::false_type{}, 0.f, 0.f, ua);
        record(a.k0 + t, P1{});
        __syncthreads();
        live = failed == 0;
        if (t + 1 == tck) {
            res_checkpoint<CPL, RPW>(a, gl, fbase, t + 1, ub, ua, lane, me.n);
            tck = res_next_checkpoint(a, t + 2);
        }
    }
    if (t == T && live) {
        step(ua, ub, t, P0{}, std::false_type{}, 0.f, 0.f, ua);
        record(a.k0 + t - 1, P0{});
        __syncthreads();
    }
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
                if (r < me.n) {
                    float* o = a.out + gl * a.outstride + (int64_t)(j0 + r) * nx;
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
    cluster_sync();
}

// A row of quotients x / HH, HH = h^2: a product with the rounded reciprocal y, its exact remainder
// and one correction, which is the correctly rounded quotient where the reciprocal is correctly
// rounded and nothing under- or overflows (P. Markstein, Computation of elementary functions on the
// IBM RISC System/6000 processor, 1990).  Ahead of a wave front the field runs through every
// magnitude down to the smallest subnormal, so the row is scaled by 2^64 first and back afterwards,
// which is exact but for quotients that are subnormal themselves, of x = 1 .. 8 x 2^-149; there the
// second rounding goes wrong for 5 and 6, by one unit, which is taken back.  Tested against division
// for every significand and in the subnormal range.  The scaled quotient is x 2^64 10^6, below 2^127 up
// to x = 2^43; a lane with a value above that divides.  (A zero keeps only its value, not its sign.)
__device__ __forceinline__ float tiny_quotient(float q, float x) {
    const uint32_t b = 2u * __float_as_uint(x);
    return b == 10u || b == 12u ? __uint_as_float(__float_as_uint(q) - 1u) : q;
}
template <int NP>
__device__ __forceinline__ void div_hh(float2 (&x)[NP]) {
    constexpr float HH = kRefH * kRefH, y = 1.0f / HH;
    float most = 0.f;
    uint32_t least = 0xffffffffu;                          // of 2 x bits - 1: a zero wraps to the largest
#pragma unroll
    for (int v = 0; v < NP; ++v) {
        most = fmaxf(most, fmaxf(fabsf(x[v].x), fabsf(x[v].y)));
        least = min(least, min(2u * __float_as_uint(x[v].x) - 1u, 2u * __float_as_uint(x[v].y) - 1u));
    }
    if (most > 0x1p43f) {
#pragma unroll
        for (int v = 0; v < NP; ++v) x[v] = make_float2(__fdiv_rn(x[v].x, HH), __fdiv_rn(x[v].y, HH));
        return;
    }
    const bool tiny = least < 16u;
#pragma unroll
    for (int v = 0; v < NP; ++v) {
        const float2 s = pk_mul(x[v], make_float2(0x1p64f, 0x1p64f)), q = pk_mul(s, make_float2(y, y));
        const float2 o = pk_mul(pk_fma(pk_fma(make_float2(-HH, -HH), q, s), make_float2(y, y), q), make_float2(0x1p-64f, 0x1p-64f));
        x[v] = tiny ? make_float2(tiny_quotient(o.x, x[v].x), tiny_quotient(o.y, x[v].y)) : o;
    }
}

// Cell i (the same in every lane) of the lanes with `on` takes its west (WEST) or east neighbour's
// value in b plus add; west, east: the lane's outer neighbours.
template <int CPL, bool WEST>
__device__ __forceinline__ void from_side(float2 (&x)[CPL / 2], const float2 (&b)[CPL / 2], int i, bool on, float west,
                                          float east, bool sensor, float add) {
#pragma unroll
    for (int k = 0; k < CPL; ++k)
        if (i == k) {
            const int n = WEST ? k - 1 : k + 1;
            float v = n < 0 ? west : n >= CPL ? east : n % 2 == 0 ? b[(n < 0 ? 0 : n) / 2 % (CPL / 2)].x : b[(n < 0 ? 0 : n) / 2 % (CPL / 2)].y;
            if (sensor) v = xa(v, add);
            float& o = k % 2 == 0 ? x[k / 2].x : x[k / 2].y;
            o = on ? v : o;
        }
}

template <int CPL, int RPW, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_ref_adj(DevGeo g, ResAdj a) {
    using F = Frag<CPL>;
    constexpr int NP = F::NP, ROW = F::ROW, D = res_depth<CPL, RPW>;
    static_assert(RPW == 2, "rows come in pairs");
    extern __shared__ __align__(1024) unsigned char smraw[];
    const int W = blockDim.x >> 5, lane = threadIdx.x & 31, w = __shfl_sync(FULL, (int)threadIdx.x >> 5, 0);
    const ResSmem sm = res_smem<CPL, RPW, false>(smraw, W);
    const int rank = (int)cluster_rank(), cs = a.cs, gl = blockIdx.x / cs;
    const int nx = g.nx, ny = g.ny, T = a.T, lo = g.lo, hi = g.hi;
    const RefRows me = ref_rows(a.warps, a.nwarps, rank * W + w);
    const int j0 = me.j0;
    const bool single = me.n == 1;
    res_setup(sm, rank, cs, 4 * ROW, 4u * ROW, a.w.extra_tx);
    ResLinks<CPL> lk;
    lk.init(sm, rank, cs, w == 0, w == W - 1, a.w.wait_ns);
    lk.single = single;
    const int64_t fbase = (int64_t)j0 * ROW;
    const float* hp = a.hist + gl * a.hstride + (int64_t)(a.kz0 - a.qlo) * a.ns + fbase;
    float* const ring = sm.ring + w * RPW * ROW;
    int left = T;
    auto request = [&](int i) {
        if (left > 0) {
#pragma unroll
            for (int r = 0; r < RPW; ++r)
                if (r < me.n) row_async<CPL>(ring + (i * W * RPW + r) * ROW, hp + r * ROW, lane);
            hp -= a.ns;
            --left;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int r = 0; r < RPW; ++r)
        if (r >= me.n) {
            const float2 none[NP] = {};
            for (int i = 0; i < D; ++i) F::store(ring + (i * W * RPW + r) * ROW, none, lane);
        }
    for (int i = 0; i < D; ++i) request(i);
    float2 of[RPW][NP], za[RPW][NP], zb[RPW][NP], pa[RPW][NP], pb[RPW][NP], co[RPW][NP];
    const float2 zero = make_float2(0.f, 0.f);
    float* const st = a.st + gl * a.ststride + fbase;
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int j = j0 + r;
        const bool in = r < me.n;
#pragma unroll
        for (int v = 0; v < NP; ++v) {
            const int x = CPL * lane + 2 * v;
            of[r][v].x = in && x < nx ? xa(1.f, a.field[(int64_t)j * nx + x]) : 0.f;
            of[r][v].y = in && x + 1 < nx ? xa(1.f, a.field[(int64_t)j * nx + x + 1]) : 0.f;
            za[r][v] = zb[r][v] = co[r][v] = zero;
        }
        if (!a.first && in) {
            F::load(za[r], st + r * ROW, lane);
            F::load(zb[r], st + a.ns + r * ROW, lane);
            F::load(co[r], st + 2 * a.ns + r * ROW, lane);
        }
#pragma unroll
        for (int v = 0; v < NP; ++v) pa[r][v] = pk_mul(of[r][v], za[r][v]);
    }
    // columns of the sensor rows among the lane's cells; lane and cell of the right edge and of the
    // sensor columns
    unsigned line = 0u;
#pragma unroll
    for (int i = 0; i < CPL; ++i)
        if (CPL * lane + i > lo && CPL * lane + i < hi) line |= 1u << i;
    const int l_e = (nx - 1) / CPL, i_e = nx - 1 - l_e * CPL, l_lo = lo / CPL, i_lo = lo - l_lo * CPL, l_hi = hi / CPL,
              i_hi = hi - l_hi * CPL;
    bool side[2];              // rows with sensor columns
    side[0] = j0 > lo && j0 < hi;
    side[1] = j0 + 1 > lo && j0 + 1 < hi && !single;
    const bool low_line = j0 == lo && !single, high_line = j0 + 1 == hi && !single;
    const bool first_row = j0 == 0, last_row = j0 == ny - 2;
    // receivers of the block in row order; the index of the lane's first in each row
    const RefRows blo = ref_rows(a.warps, a.nwarps, rank * W), bhi = ref_rows(a.warps, a.nwarps, min(rank * W + W, a.nwarps) - 1);
    const int n0 = a.rowstart[blo.j0], n1 = a.rowstart[bhi.j0 + bhi.n], nrec = n1 - n0;
    int rb[2];
    rb[0] = rb[1] = 0;
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        const int j = j0 + r;
        if (r >= me.n) continue;
        const int f = a.rowstart[j] - n0;
        rb[r] = j == lo || j == hi ? f + max(0, CPL * lane - (lo + 1)) : f;   // columns lo+1 .. hi-1; lo and hi
    }
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
    auto inject = [](float v) { return xm(xm(v, kRefH), 1000.f); };   // (rr H) 1000
    auto stage = [&](int t, auto pc, float v) {
        constexpr int P = decltype(pc)::value;
        if (stg) sm.val[P * nrec + ri] = inject(v);
        if (stg_more && t <= T)
            for (int n = ri + blockDim.x; n < nrec; n += blockDim.x)
                sm.val[P * nrec + n] = inject(rr[(int64_t)(a.kz0 - t + 1) * g.nch + a.rchan[n0 + n]]);
    };
    using P0 = std::integral_constant<int, 0>;
    using P1 = std::integral_constant<int, 1>;
    float rv0 = 0.f, rv1 = 0.f;
    next_res(rv1);
    stage(1, P1{}, rv1);
    next_res(rv0);
    next_res(rv1);
    float* const xw = sm.xch + w * RPW * 2 * ROW;
    auto publish = [&](const float2 (&x)[RPW][NP], auto pc) {
        constexpr int P = decltype(pc)::value;
        F::store(xw + P * ROW, x[0], lane);
        if (single) F::store(xw + (2 + P) * ROW, x[0], lane);
        else F::store(xw + (2 + P) * ROW, x[1], lane);
        lk.template send<P>(x[0], x[1], lane);
    };
    __syncthreads();
    cluster_sync();
    publish(pa, P0{});
    __syncthreads();

    const float* const srow = w > 0 ? xw - 2 * ROW : sm.halo;
    const float* const nrow = w < W - 1 ? xw + RPW * 2 * ROW : sm.halo + 2 * ROW;
    constexpr float A = (1500.f * 1500.f) * (kRefDT * kRefDT);
    const float2 A2 = make_float2(A, A);
    int hi_slot = 0;
    auto step = [&](float2 (&zc)[RPW][NP], float2 (&zp)[RPW][NP], float2 (&pc)[RPW][NP], float2 (&pn)[RPW][NP], int t,
                    auto par) {
        constexpr int P = decltype(par)::value;
        lk.template recv<P>(sm, t, lane);
        const float* const vals = sm.val + (P ^ 1) * nrec;
        float2 sb[NP], nb[NP];
        F::load(sb, srow + P * ROW, lane);
        F::load(nb, nrow + P * ROW, lane);
        if (single) {
#pragma unroll
            for (int v = 0; v < NP; ++v) pc[1][v] = nb[v];
        }
        // backpropagation1 on every cell
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const float wl = __shfl_up_sync(FULL, pc[r][NP - 1].y, 1), er = __shfl_down_sync(FULL, pc[r][0].x, 1);
            float2 x[NP];
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                const float2 q = pc[r][v];
                const float2 sn = pk_add(r == 0 ? sb[v] : pc[0][v], r == 1 ? nb[v] : pc[1][v]);
                const float we = v > 0 ? pc[r][v - 1].y : wl, ee = v + 1 < NP ? pc[r][v + 1].x : er;
                const float2 l = pk_fma(make_float2(-4.f, -4.f), q, make_float2(xa(xa(sn.x, we), q.y), xa(xa(sn.y, q.x), ee)));
                x[v] = mul2(A2, l);
            }
            div_hh(x);
#pragma unroll
            for (int v = 0; v < NP; ++v) zp[r][v] = pk_sub(pk_add(x[v], pk_add(zc[r][v], zc[r][v])), zp[r][v]);
        }
        if (single) {
#pragma unroll
            for (int v = 0; v < NP; ++v) zp[1][v] = zero;
        }
        // sensor rows: the inner row's value plus the residual; before that row's own sensor columns
        if (low_line) {
            int b = rb[0];
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                if ((line >> (2 * v)) & 1u) zp[0][v].x = xa(zp[1][v].x, vals[b++]);
                if ((line >> (2 * v)) & 2u) zp[0][v].y = xa(zp[1][v].y, vals[b++]);
            }
        }
        if (high_line) {
            int b = rb[1];
#pragma unroll
            for (int v = 0; v < NP; ++v) {
                if ((line >> (2 * v)) & 1u) zp[1][v].x = xa(zp[0][v].x, vals[b++]);
                if ((line >> (2 * v)) & 2u) zp[1][v].y = xa(zp[0][v].y, vals[b++]);
            }
        }
        // edge and sensor columns: the inner neighbour's value (plus the residual)
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const float wl = __shfl_up_sync(FULL, zp[r][NP - 1].y, 1), er = __shfl_down_sync(FULL, zp[r][0].x, 1);
            float2 b[NP];
#pragma unroll
            for (int v = 0; v < NP; ++v) b[v] = zp[r][v];
            if (side[r]) {
                from_side<CPL, false>(zp[r], b, i_lo, lane == l_lo, wl, er, true, vals[rb[r]]);
                from_side<CPL, true>(zp[r], b, i_hi, lane == l_hi, wl, er, true, vals[rb[r] + 1]);
            }
            from_side<CPL, true>(zp[r], b, i_e, lane == l_e, wl, er, false, 0.f);
            if (lane == 0) zp[r][0].x = b[0].y;
        }
        __syncwarp();
        if (first_row) {
#pragma unroll
            for (int v = 0; v < NP; ++v) zp[0][v] = zp[1][v];
        }
        if (last_row) {
#pragma unroll
            for (int v = 0; v < NP; ++v) zp[1][v] = zp[0][v];
        }
#pragma unroll
        for (int r = 0; r < RPW; ++r)
#pragma unroll
            for (int v = 0; v < NP; ++v) pn[r][v] = pk_mul(of[r][v], zp[r][v]);
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
            F::load(lu, ring + (hi_slot * W * RPW + r) * ROW, lane);
#pragma unroll
            for (int v = 0; v < NP; ++v) co[r][v] = pk_fma(zp[r][v], lu[v], co[r][v]);
        }
        request(hi_slot);
        if (D > 1) hi_slot = hi_slot + 1 == D ? 0 : hi_slot + 1;
        __syncthreads();
    };
    bool live = true;
#pragma unroll 1
    for (int t = 1; t <= T && live; t += 2) {
        const int failed = res_failed(sm, t);
        step(za, zb, pa, pb, t, P0{});
        if (t == T) break;
        step(zb, za, pb, pa, t + 1, P1{});
        live = failed == 0;
    }
    if (live) {
        if (T & 1) lk.template recv<1, false>(sm, T + 1, lane);
        else lk.template recv<0, false>(sm, T + 1, lane);
    }
    __syncthreads();
    if (*sm.bad == 0) {
        const bool odd = T & 1;
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            if (r >= me.n) continue;
            if (a.last) {
                F::store_nat(a.corr + gl * a.cstride + (int64_t)(j0 + r) * nx, co[r], lane, nx);
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
template <int CPL, typename Args>
cudaError_t ref_go(const ResShape& s, const DevGeo* g, const Args* a, int* held, void* stream) {
    constexpr bool fwd = std::is_same<Args, ResFwd>::value;
    // the forward sweep's two edge rows, the adjoint's two steps of residuals
    const size_t smem = res_smem_bytes<CPL, 2>(s.warps, fwd, s.nrec) + (fwd ? 8 * (size_t)Frag<CPL>::ROW : 0);
    if (s.warps > 8) {
        if constexpr (fwd) return res_call(k_ref_fwd<CPL, 2, 512>, s, smem, g, a, held, stream);
        else return res_call(k_ref_adj<CPL, 2, 512>, s, smem, g, a, held, stream);
    }
    if constexpr (fwd) return res_call(k_ref_fwd<CPL, 2, 256>, s, smem, g, a, held, stream);
    else return res_call(k_ref_adj<CPL, 2, 256>, s, smem, g, a, held, stream);
}

}  // namespace
}  // namespace tomo
