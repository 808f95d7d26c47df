// fluidx and advectbyzx of the x sweep (FP32) for pencil lengths that the fixed-length
// register engines (mhd_fluidx2.cuh, mhd_advect2/3/6.cuh) were not laid out for (100,
// 72, 75 cells), and for arrays that are not 16-byte aligned; short pencils and small
// boxes of them take one thread per cell (thread_per_cell_fluidx, _advect in
// kernels_impl.cuh).  EXACT gives the oracle's bits; FAST those of the one-thread-per-cell
// kernels, which the tests pin.
//
// A pencil of n cells is held by T = ceil(n / C) threads with C (3, 4 or 5)
// consecutive cells in registers; the last one holds the remaining L cells and,
// in its other C - L slots, periodic images of cells 0 .. C-L-1, so no exchange
// is special but for its two ends: thread 0 sends its cell C-L backwards
// instead of its cell 0, and the last thread sends its cell L-1 forwards.  A group of
// G = 8, 16 or 32 W lanes holds a pencil (G >= T; the lanes past T repeat the
// last thread and write nothing); C is the one with the fewest slots G C.
// Up to 160 cells fluidx needs no barrier of its own: all exchanges are shuffles.
// Longer pencils cross warps through shared memory and the CTA barrier.  advectbyzx looks
// two cells ahead, so its last thread holds two at least: 101, 131, 136, 141, 146, 151 and
// 156 cells cross warps too, and a length one above a multiple of 60 has no such layout (k_advect).
//
// A pencil is staged by one bulk copy where it consists of aligned 16-byte
// pieces, by 8- or 4-byte cp.async otherwise; the images are staged as well.  The kernels this
// replaced took one thread per cell and exchanged through shared memory, with a
// CTA barrier for every step of the stencil.  Both are bound by instruction
// issue and latency (the boxes fit in L2).
//
// Measured (plain steps, with the transposes of mhd_kernels.cuh): four steps of
// 100 x 72 x 72 in 1.67 ms with one thread per cell, 0.95 ms; one step of 200 x 150 x 150 1.34 ms.
#pragma once
#include "mhd_kernels.cuh"
#include "mhd_launch.h"
#include "mhd_pencil.cuh"

namespace mhd {

constexpr int kRagThreads = 128;                 // threads per fluidx CTA (at least one pencil)
constexpr int kRagSeam = 2 * 16 * kSeamVals;     // two banks, up to 16 warps
__host__ __device__ inline int rag_up4(int x) { return (x + 3) & ~3; }

// pencils per CTA
inline int rag_pencils(const RagShape& s) { return s.G >= kRagThreads ? 1 : kRagThreads / s.G; }

inline size_t rag_fluidx_smem(const RagShape& s)
{
    const int P = rag_pencils(s), tc = s.T * s.C;
    return ((size_t)P * rag_up4(5 * tc) + (size_t)(2 * P + 1) * rag_up4(3 * tc) + 32 + kRagSeam) * sizeof(float);
}

// slots of one advectbyzx plane: J+2 pencils of (rho, m_x), J+1 of b
inline size_t rag_advect_smem(const RagShape& s, int J)
{
    const int tc = s.T * s.C;
    return ((size_t)2 * ((J + 2) * rag_up4(2 * tc) + (J + 1) * rag_up4(3 * tc)) + (size_t)2 * (J + 1) * rag_up4(tc) +
            kRagSeam) * sizeof(float);
}

// The exchanges of one pencil's group.
template <int C, int D>
struct RagGroup {
    static constexpr int L = C - D;  // cells of the last thread
    int T, G, t, lane, warp, gw0, nw;  // threads, lanes; thread, first warp, warps
    bool last, real;

    __device__ __forceinline__ RagGroup(const RagShape& s, int tid)
    {
        T = s.T;
        G = s.G;
        lane = tid & 31;
        warp = tid >> 5;
        const int r = (G <= 32) ? (tid & (G - 1)) : tid % G;
        real = r < T;
        t = real ? r : T - 1;
        last = (t == T - 1);
        nw = (G + 31) >> 5;
        gw0 = warp - (G > 32 ? (r >> 5) : 0);
    }
    __device__ __forceinline__ bool multi() const { return G > 32; }
    // The CTA barrier: every group of a CTA makes the same calls.  (A named barrier
    // per group with a run-time index reserves all 16 of them for each CTA, which
    // leaves four CTAs on an SM.)
    __device__ __forceinline__ void sync() const { __syncthreads(); }
    // cells of this thread that are its own (the others are images or repeats)
    __device__ __forceinline__ int own() const { return real ? (last ? L : C) : 0; }

    __device__ __forceinline__ float max(float x, float* red) const
    {
        if (!multi()) {
            for (int o = G / 2; o > 0; o >>= 1)
                x = fmaxf(x, __shfl_xor_sync(kFull, x, o));
            return fmaxf(0.f, x);
        }
        x = real ? x : 0.f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            x = fmaxf(x, __shfl_xor_sync(kFull, x, o));
        if (lane == 0)
            red[warp] = x;
        sync();
        float m = 0.f;
        for (int s = 0; s < nw; s++)
            m = fmaxf(m, red[gw0 + s]);
        return m;
    }

    // out[k] = x[k] of the next (dir +1) or the previous (dir -1) thread of the pencil
    template <int K>
    __device__ __forceinline__ void move(const float (&x)[K], float (&out)[K], int dir, float* seam, int bank) const
    {
        if (!multi()) {
            const int src = (dir > 0) ? (last ? 0 : t + 1) : (t == 0 ? T - 1 : t - 1);
#pragma unroll
            for (int k = 0; k < K; k++)
                out[k] = __shfl_sync(kFull, x[k], src, G);
            return;
        }
        float* s = seam + bank * (16 * kSeamVals);
        if (dir > 0 ? lane == 0 : (real && (last || lane == 31))) {
#pragma unroll
            for (int k = 0; k < K; k++)
                s[warp * kSeamVals + k] = x[k];
        }
#pragma unroll
        for (int k = 0; k < K; k++)
            out[k] = (dir > 0) ? __shfl_down_sync(kFull, x[k], 1) : __shfl_up_sync(kFull, x[k], 1);
        sync();
        if (dir > 0 ? (last || lane == 31) : lane == 0) {
            const int from = (dir > 0) ? (last ? gw0 : warp + 1) : (t == 0 ? gw0 + nw - 1 : warp - 1);
#pragma unroll
            for (int k = 0; k < K; k++)
                out[k] = s[from * kSeamVals + k];
        }
    }

    // the N cells after this thread's (x[m] of cell m of C, K values a cell)
    template <int K, int N>
    __device__ __forceinline__ void next(const float (&x)[C][K], float (&out)[N][K], float* seam, int bank) const
    {
        float v[N * K], r[N * K];
#pragma unroll
        for (int m = 0; m < N; m++)
#pragma unroll
            for (int k = 0; k < K; k++)
                v[m * K + k] = x[m][k];
        if (D > 0 && t == 0) {  // its receiver, the last thread, holds cells 0 .. D-1 as images
#pragma unroll
            for (int m = 0; m < N; m++)
#pragma unroll
                for (int k = 0; k < K; k++)
                    v[m * K + k] = x[D + m < C ? D + m : C - 1][k];  // D + m < C by the choice of C (or n = 1)
        }
        move<N * K>(v, r, +1, seam, bank);
#pragma unroll
        for (int m = 0; m < N; m++)
#pragma unroll
            for (int k = 0; k < K; k++)
                out[m][k] = r[m * K + k];
    }

    // the cell before this thread's
    template <int K>
    __device__ __forceinline__ void prev(const float (&x)[C][K], float (&out)[K], float* seam, int bank) const
    {
        float v[K];
#pragma unroll
        for (int k = 0; k < K; k++)
            v[k] = x[C - 1][k];
        if (D > 0 && last) {
#pragma unroll
            for (int k = 0; k < K; k++)
                v[k] = x[L - 1][k];
        }
        move<K>(v, out, -1, seam, bank);
    }
};

// `rows` pencils of NC words a cell into shared memory at a stride of DS words,
// the images of cells 0 .. tc-n-1 after cell n-1; a warp takes whole pencils
// (from row `first` on, every `nw`-th).  src(row) is the pencil's first word in
// global memory, SC words a cell (its first NC are taken).  pb: bytes of the
// pieces that pencils consist of: 16 (one bulk copy a pencil, completing on
// `bar`, whose expected bytes the caller has set), 8 or 4 (cp.async).
template <int NC, int SC, typename Src>
__device__ __forceinline__ void rag_stage(float* dst, int DS, int rows, int n, int tc, int pb, Src src, int first, int nw,
                                          int lane, uint64_t* bar)
{
    for (int r = first; r < rows; r += nw) {
        const float* s = src(r);
        float* d = dst + r * DS;
        if (SC == NC && pb == 16) {
            if (lane == 0)
                tma_load_1d(d, s, (uint32_t)(n * NC * 4), bar);
        } else if (SC == NC && pb == 8) {
#pragma unroll 4
            for (int w = lane; w < n * NC / 2; w += 32)
                cp_async8(d + 2 * w, s + 2 * w);
        } else if (SC == NC) {
#pragma unroll 4
            for (int w = lane; w < n * NC; w += 32)
                cp_async4(d + w, s + w);
        } else {
#pragma unroll 4
            for (int c = lane; c < n; c += 32)
#pragma unroll
                for (int q = 0; q < NC; q++)
                    cp_async4(d + NC * c + q, s + SC * c + q);
        }
        if (lane < tc - n) {  // images
#pragma unroll
            for (int q = 0; q < NC; q++)
                cp_async4(d + NC * (n + lane) + q, s + SC * (lane % n) + q);
        }
    }
}

// NF consecutive words of shared memory: 16 bytes at a time when C = 4
template <int C, int NF>
__device__ __forceinline__ void rag_lds(const float* s, float (&d)[NF])
{
    if constexpr (C == 4) {
        lds_chunk<float, NF>(s, d);
    } else {
#pragma unroll
        for (int v = 0; v < NF; v++)
            d[v] = s[v];
    }
}

// CTAs per SM that k_fluidx_rag is bounded to in FAST (0: as the compiler finds): five (96
// registers, C = 3: seven and 72) for the kinds that hold in it without spills but take 128 or 79
// without a bound (pencils of 72 cells, four CTAs instead of five: 14.6 against 10.6 us); four
// for <4, 3>, which takes 96 by itself and is faster with 128 (121 and 241 cells: 4 to 8%).
constexpr int rag_fluidx_ctas(int C, int D)
{
    return C == 3 ? (D == 2 ? 7 : 0) : (C == 5 ? (D >= 3 ? 5 : 0) : (D % 3 ? 5 : (D == 3 ? 4 : 0)));
}

// C/fluidx.c:19-102, C/tvd1.c:8-118, C/mhdflux.c:9-72; see fluidx2_body for the
// arithmetic, which this repeats expression by expression.
template <bool EX, int C, int D>
__global__ void __launch_bounds__(kRagThreads, EX ? 0 : rag_fluidx_ctas(C, D)) k_fluidx_rag(FluidxArgs a, RagShape sh, int pb)
{
    after_previous();
    using R = float;
    select_box(a, blockIdx.z, sizeof(CflPart<R>), gridDim.x * gridDim.y);
    extern __shared__ __align__(16) float rag_smem[];
    const int n = a.nx, P = a.P, tid = threadIdx.x, tc = sh.T * C;
    const RagGroup<C, D> g(sh, tid);
    const int j0 = blockIdx.x * P, k = blockIdx.y, kp = (k + 1 == a.nz) ? 0 : k + 1;
    const int np = min(P, a.ny - j0);              // pencils of this CTA
    const int lp = min(tid / sh.G, np - 1);        // groups past np repeat the last pencil
    const bool live = tid / sh.G < np;
    const int i0 = g.t * C, own = live ? g.own() : 0;
    const int SU = rag_up4(5 * tc), SB = rag_up4(3 * tc);
    float* const su = rag_smem;
    float* const sb = su + P * SU;         // pencils j0 .. j0+np
    float* const sbk = sb + (P + 1) * SB;  // plane kp; then the cell-centred field of this thread's cells
    float* const red = sbk + P * SB;
    float* const seam = red + 32;
    const R* uu = static_cast<const R*>(a.uu);
    const R* ub = static_cast<const R*>(a.ub);
    const size_t c0 = ((size_t)k * a.ny + j0) * n;
    __shared__ uint64_t bar;
    const int lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    if (pb == 16) {
        if (tid == 0) {
            mbar_init(&bar, 1);
            mbar_arrive_expect_tx(&bar, (uint32_t)(np * n * 20 + (2 * np + 1) * n * 12));
        }
        __syncthreads();
    }
    // the three arrays' pencils dealt over the warps in one round
    rag_stage<5, 5>(su, SU, np, n, tc, pb, [&](int r) { return uu + (c0 + (size_t)r * n) * 5; }, wid, nw, lane, &bar);
    rag_stage<3, 3>(sb, SB, np + 1, n, tc, pb, [&](int r) {
        const int j = (j0 + r == a.ny) ? 0 : j0 + r;
        return ub + ((size_t)k * a.ny + j) * n * 3;
    }, (wid + nw - np % nw) % nw, nw, lane, &bar);
    rag_stage<3, 3>(sbk, SB, np, n, tc, pb, [&](int r) { return ub + ((size_t)kp * a.ny + j0 + r) * n * 3; },
                    (wid + nw - (2 * np + 1) % nw) % nw, nw, lane, &bar);
    const R dt = load_dt<R>(a.dt_ptr, a.dt_val);
    cp_async_commit();
    cp_async_wait<0>();
    // a bulk copy that never lands: the CTA leaves before computing (error bit set)
    if (!__syncthreads_and(pb != 16 || mbar_wait_bounded(&bar, 0, a.err)))
        return;

    R* const uq = su + lp * SU + i0 * 5;
    R* const fown = sbk + lp * SB + i0 * 3;
    auto load_q = [&](R (&q)[C][5]) {
        R t[C * 5];
        rag_lds<C, C * 5>(uq, t);
#pragma unroll
        for (int m = 0; m < C; m++)
#pragma unroll
            for (int s = 0; s < 5; s++)
                q[m][s] = t[5 * m + s];
    };
    R q[C][5], f[C][3];
    load_q(q);
    {
        R bj[C * 3], bp[C * 3], bk[C * 3];
        const R* row = sb + lp * SB;
        rag_lds<C, C * 3>(row + 3 * i0, bj);
        rag_lds<C, C * 3>(row + SB + 3 * i0, bp);
        rag_lds<C, C * 3>(fown, bk);
        const R b1next = row[3 * (g.last ? tc % n : i0 + C)];
#pragma unroll
        for (int m = 0; m < C; m++) {
            const R b0n = (m + 1 < C) ? bj[3 * (m + 1)] : b1next;
            f[m][0] = R(0.5) * bj[3 * m] + R(0.5) * b0n;
            f[m][1] = R(0.5) * bj[3 * m + 1] + bp[3 * m + 1] / R(2);
            f[m][2] = R(0.5) * bj[3 * m + 2] + bk[3 * m + 2] / R(2);
        }
    }

    // fluxes of the state w: fr = c (w + v / c), gl = c (w - v / c) (C/tvd1.c:33-49, 51-69).
    // (FAST: the expressions of k_fluidx, which the compiler contracts alike)
    R fr[C][5], gl[C][5];
    auto fluxes = [&](const R (&w)[C][5], R* rd) {
        R v[C][5], cm = R(0);
#pragma unroll
        for (int m = 0; m < C; m++) {
            R ci;
            if constexpr (EX)
                cell_flux<R, EX>(w[m], f[m], v[m], ci);
            else
                cell_flux_pinned(w[m], f[m], v[m], ci);
            cm = fmaxf(cm, ci);
        }
        const R c = g.max(cm, rd);
#pragma unroll
        for (int m = 0; m < C; m++) {
            scale_flux<R, EX>(v[m], c);
#pragma unroll
            for (int s = 0; s < 5; s++) {
                fr[m][s] = scale0<R, EX>(c, lin<R, EX>(R(1), w[m][s], R(1), v[m][s]));
                gl[m][s] = scale0<R, EX>(c, lin<R, EX>(R(1), w[m][s], R(-1), v[m][s]));
            }
        }
    };
    // w + h (F(i) - F(i-1)) into q
    R flux[C][5];
    auto update = [&](R (&w)[C][5], R h) {
        R fp[5];
        g.template prev<5>(flux, fp, seam, 1);
#pragma unroll
        for (int m = 0; m < C; m++)
#pragma unroll
            for (int s = 0; s < 5; s++)
                w[m][s] = lin<R, EX>(R(1), w[m][s], h,
                                     lin<R, EX>(R(1), flux[m][s], R(-1), (m > 0) ? flux[m - 1][s] : fp[s]));
    };

    // ---- stage 1
    fluxes(q, red);
    {
        R gn[1][5];
        g.template next<5, 1>(gl, gn, seam, 0);
#pragma unroll
        for (int m = 0; m < C; m++)
#pragma unroll
            for (int s = 0; s < 5; s++) {
                const R x = (m + 1 < C) ? gl[m + 1][s] : gn[0][s];
                flux[m][s] = lin<R, EX>(R(0.5), fr[m][s], R(-0.5), x);
            }
        update(q, R(-0.5) * dt);
    }
    // ---- stage 2
    fluxes(q, red + 16);
    {
        R frp[5], gn[1][5], d[C][10], dn[1][10];
        g.template prev<5>(fr, frp, seam, 0);
        g.template next<5, 1>(gl, gn, seam, 1);
#pragma unroll
        for (int m = 0; m < C; m++)
#pragma unroll
            for (int s = 0; s < 5; s++) {
                const R p = (m > 0) ? fr[m - 1][s] : frp[s], x = (m + 1 < C) ? gl[m + 1][s] : gn[0][s];
                d[m][s] = lin<R, EX>(R(0.5), fr[m][s], R(-0.5), p);
                d[m][5 + s] = lin<R, EX>(R(0.5), gl[m][s], R(-0.5), x);
            }
        g.template next<10, 1>(d, dn, seam, 0);
#pragma unroll
        for (int m = 0; m < C; m++)
#pragma unroll
            for (int s = 0; s < 5; s++) {
                const R dr = (m + 1 < C) ? d[m + 1][s] : dn[0][s], dl = (m + 1 < C) ? d[m + 1][5 + s] : dn[0][5 + s];
                const R x = (m + 1 < C) ? gl[m + 1][s] : gn[0][s];
                const R a1 = vanleer<R, EX>(dr, d[m][s]), a2 = vanleer<R, EX>(dl, d[m][5 + s]);
                flux[m][s] = lin<R, EX>(R(0.5), lin<R, EX>(R(1), fr[m][s], R(-1), x), R(0.5),
                                        lin<R, EX>(R(1), a1, R(-1), a2));
            }
        load_q(q);
        update(q, -dt);
    }
#pragma unroll
    for (int m = 0; m < C; m++)
        if (m < own) {
#pragma unroll
            for (int s = 0; s < 5; s++)
                uq[5 * m + s] = q[m][s];  // no other thread reads this thread's cells (images are copies)
            if (a.w_out) {
                const size_t cell = c0 + (size_t)lp * n + i0 + m;
                reinterpret_cast<float2*>(a.w_out)[cell] = make_float2(q[m][0], q[m][1]);
            }
        }

    before_next();
    // ---- optional calcfl epilogue on the new state (face b at (j,k))
    if (a.cfl_part) {
        const R* bj = sb + lp * SB + 3 * i0;
        R mx = R(0);
        int ln = -1;
#pragma unroll
        for (int m = 0; m < C; m++)
            if (m < own) {
                const R fc[3] = {bj[3 * m], bj[3 * m + 1], bj[3 * m + 2]};
                const R sp = cfl_speed<R, EX>(q[m], fc);
                if (sp != sp)
                    ln = (int)(c0 + (size_t)lp * n + i0 + m);
                else
                    mx = fmaxf(mx, sp);
            }
        mx = warp_max<R>(mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            ln = max(ln, __shfl_xor_sync(kFull, ln, o));
        __syncthreads();  // red and seam are reused below
        int* rn = reinterpret_cast<int*>(seam);
        if ((tid & 31) == 0) {
            red[tid >> 5] = mx;
            rn[tid >> 5] = ln;
        }
        __syncthreads();
        if (tid == 0) {
            R cm = R(0);
            int lnan = -1;
            for (int s = 0; s < (int)(blockDim.x >> 5); s++) {
                cm = fmaxf(cm, red[s]);
                lnan = max(lnan, rn[s]);
            }
            CflPart<R>* part = static_cast<CflPart<R>*>(a.cfl_part) + ((size_t)k * gridDim.x + blockIdx.x);
            part->cmax = cm;
            part->last_nan = lnan;
        }
    }
    R* uo = static_cast<R*>(a.u_out) + c0 * 5;
    if (pb == 16) {
        fence_proxy_async_smem();
        __syncthreads();
        if (tid == 0) {
            for (int r = 0; r < np; r++)
                tma_store_1d(uo + (size_t)r * n * 5, su + r * SU, (uint32_t)(n * 20));
            tma_store_commit();
            tma_store_wait_read();
        }
        return;
    }
    __syncthreads();
    for (int r = wid; r < np; r += nw) {
        R* d = uo + (size_t)r * n * 5;
        const R* t = su + r * SU;
        if (pb == 8) {
            for (int w = lane; w < n * 5 / 2; w += 32)
                reinterpret_cast<float2*>(d)[w] = reinterpret_cast<const float2*>(t)[w];
        } else {
            for (int w = lane; w < n * 5; w += 32)
                d[w] = t[w];
        }
    }
}

// Half step of tvdb, in both policies with the reference's roundings: the product, then
// b - x / 2 once (FAST: the bits of k_advect, the kernel of these lengths before).
__device__ __forceinline__ float rag_half(float bv, float f1, float fm, float dt)
{
    return __fmaf_rn(-0.5f, __fmul_rn(__fsub_rn(f1, fm), dt), bv);
}

// One tvdb row of a group, as tvdb_row (mhd_advect2.cuh) for these groups.
template <bool EX, int C, int D>
__device__ __forceinline__ void rag_tvdb_row(const RagGroup<C, D>& g, const float (&vr)[C][1], const float (&bv)[C],
                                             float dt, float* seam, float (&F)[C], float (&bnew)[C])
{
    float t[C][2];  // vg, b vg
    {
        float l[1], r[1][1];
        g.template prev<1>(vr, l, seam, 0);
        g.template next<1, 1>(vr, r, seam, 1);
#pragma unroll
        for (int m = 0; m < C; m++) {
            t[m][0] = tvdb_smooth<float, EX>(m > 0 ? vr[m - 1][0] : l[0], vr[m][0], m + 1 < C ? vr[m + 1][0] : r[0][0]);
            t[m][1] = tvdb_prod<float, EX>(bv[m], t[m][0]);
        }
    }
    float vh[C], x[C][1];
    {
        float r[1][2], l[1];
        g.template next<2, 1>(t, r, seam, 0);
#pragma unroll
        for (int m = 0; m < C; m++) {
            vh[m] = tvdb_vh<float, EX>(t[m][0], m + 1 < C ? t[m + 1][0] : r[0][0]);
            x[m][0] = (vh[m] > 0.f) ? t[m][1] : (m + 1 < C ? t[m + 1][1] : r[0][1]);
        }
        g.template prev<1>(x, l, seam, 1);
        float vb[C];
#pragma unroll
        for (int m = 0; m < C; m++)
            vb[m] = tvdb_prod<float, EX>(t[m][0], rag_half(bv[m], x[m][0], m > 0 ? x[m - 1][0] : l[0], dt));
#pragma unroll
        for (int m = 0; m < C; m++)
            x[m][0] = vb[m];
    }
    {
        float l[1], r[2][1], fl[C][1];
        g.template prev<1>(x, l, seam, 0);
        g.template next<1, 2>(x, r, seam, 1);
#pragma unroll
        for (int m = 0; m < C; m++)
            fl[m][0] = tvdb_flux<float, EX>(m > 0 ? x[m - 1][0] : l[0], x[m][0], m + 1 < C ? x[m + 1][0] : r[0][0],
                                            m + 2 < C ? x[m + 2][0] : (m + 2 == C ? r[0][0] : r[1][0]), vh[m], dt);
        g.template prev<1>(fl, l, seam, 0);
#pragma unroll
        for (int m = 0; m < C; m++) {
            F[m] = m > 0 ? fl[m - 1][0] : l[0];
            bnew[m] = tvdb_new<float, EX>(bv[m], fl[m][0], F[m]);
        }
    }
}

// advectbyzx (C/advectbyzx.c:14-23): the marching scheme of mhd_advect6.cuh with
// these groups.  J pencils per CTA and one group more for the A row of the
// pencil after them, K planes; plane k+1 is staged while plane k is computed (two
// slots); what plane k+1 needs of plane k is carried in registers.  WU: (rho, m_x)
// from the side array.
template <bool EX, int C, int D, bool WU>
__global__ void __launch_bounds__(512) k_advect_rag(AdvectArgs a, RagShape sh, int pb)
{
    after_previous();
    select_box(a, blockIdx.z);
    extern __shared__ __align__(16) float rag_smem[];
    const int n = a.nx, ny = a.ny, nz = a.nz, J = a.P, tid = threadIdx.x, tc = sh.T * C;
    const RagGroup<C, D> g(sh, tid);
    const int j0 = blockIdx.x * J, k0 = blockIdx.y * a.K, k1 = min(k0 + a.K, nz);
    const int np = min(J, ny - j0), w = min(tid / sh.G, np);  // the group's pencil; np: the halo pencil
    const bool owner = tid / sh.G < np;
    const int SU = rag_up4(2 * tc), SB = rag_up4(3 * tc), SF = rag_up4(tc);
    float* const Us = rag_smem;                            // [2][J+2][SU]: pencils j0-1 .. j0+np
    float* const Bs = Us + 2 * (J + 2) * SU;               // [2][J+1][SB]: pencils j0 .. j0+np
    float* const FAx = Bs + 2 * (J + 1) * SB;              // [2][J+1][SF]
    float* const seam = FAx + 2 * (J + 1) * SF;
    const float dt = load_dt<float>(a.dt_ptr, a.dt_val);
    const float* us = static_cast<const float*>(WU ? a.w : a.uu);
    const float* ub = static_cast<const float*>(a.ub);
    const float* b1s = static_cast<const float*>(a.b1_src);
    float* bo = static_cast<float*>(a.b_out);
    constexpr int UC = WU ? 2 : 5;

    __shared__ uint64_t bar[2];
    const int lane = tid & 31, wid = tid >> 5, nw = blockDim.x >> 5;
    auto slot = [&](int p) { return (p - k0 + 1) & 1; };
    auto issue = [&](int p) {
        if (p <= k1) {
            const int s = slot(p), pp = (p < 0) ? p + nz : (p >= nz ? p - nz : p);
            rag_stage<2, UC>(Us + s * (J + 2) * SU, SU, np + 2, n, tc, pb, [&](int r) {
                int j = j0 - 1 + r;
                j = (j < 0) ? j + ny : (j >= ny ? j - ny : j);
                return us + ((size_t)pp * ny + j) * n * UC;
            }, wid, nw, lane, &bar[s]);
            rag_stage<3, 3>(Bs + s * (J + 1) * SB, SB, np + 1, n, tc, pb, [&](int r) {
                const int j = (j0 + r >= ny) ? j0 + r - ny : j0 + r;
                return ub + ((size_t)pp * ny + j) * n * 3;
            }, (wid + nw - (np + 2) % nw) % nw, nw, lane, &bar[s]);
        }
        cp_async_commit();
    };
    // the bytes of the bulk copies of plane p (by one thread, before a barrier that every issue(p) follows)
    auto expect = [&](int p) {
        if (pb == 16 && tid == 0 && p <= k1)
            mbar_arrive_expect_tx(&bar[slot(p)], (uint32_t)((WU ? (np + 2) * n * 8 : 0) + (np + 1) * n * 12));
    };
    auto landed = [&](int p) { return pb != 16 || mbar_wait_bounded(&bar[slot(p)], ((p - k0 + 1) >> 1) & 1, a.err); };
    const int i0 = g.t * C, own = owner ? g.own() : 0;
    auto u_read = [&](int s, int r, float (&rho)[C], float (&mx)[C]) {
        float t[2 * C];
        rag_lds<C, 2 * C>(Us + (s * (J + 2) + r) * SU + 2 * i0, t);
#pragma unroll
        for (int m = 0; m < C; m++) {
            rho[m] = t[2 * m];
            mx[m] = t[2 * m + 1];
        }
    };
    auto b_read = [&](int s, float (&bb)[3 * C]) { rag_lds<C, 3 * C>(Bs + (s * (J + 1) + w) * SB + 3 * i0, bb); };
    auto face = [&](const float (&rl)[C], const float (&ml)[C], const float (&rc)[C], const float (&mc)[C],
                    float (&v)[C][1]) {
#pragma unroll
        for (int m = 0; m < C; m++)
            v[m][0] = __fdiv_rn(__fadd_rn(ml[m], mc[m]), __fadd_rn(rl[m], rc[m]));
    };

    if (pb == 16 && tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
    }
    expect(k0 - 1);
    expect(k0);
    __syncthreads();
    issue(k0 - 1);
    issue(k0);
    cp_async_wait<0>();
    landed(k0 - 1);  // a bulk copy that never lands sets the error bit; the march goes on, so none is left in flight
    landed(k0);
    __syncthreads();
    float vA[C][1], b2c[C], b1c[C], rB[C], mB[C], FBc[C], b3c[C];
    {
        const int sm = slot(k0 - 1), sc = slot(k0);
        float rl[C], ml[C], rp[C], mp[C], bb[3 * C], vB[C][1], b3[C];
        u_read(sc, w, rl, ml);
        u_read(sc, w + 1, rB, mB);
        face(rl, ml, rB, mB, vA);
        b_read(sc, bb);
#pragma unroll
        for (int m = 0; m < C; m++) {
            b1c[m] = bb[3 * m];
            b2c[m] = bb[3 * m + 1];
            b3[m] = bb[3 * m + 2];
        }
        u_read(sm, w + 1, rp, mp);
        face(rp, mp, rB, mB, vB);
        rag_tvdb_row<EX, C, D>(g, vB, b3, dt, seam, FBc, b3c);
    }
    expect(k0 + 1);
    expect(k0 + 2);
    fence_proxy_async_smem();  // the slots' reads before the copies into them
    __syncthreads();
    issue(k0 + 1);
    issue(k0 + 2);
    for (int k = k0; k < k1; k++) {
        float* const fax = FAx + (k & 1) * (J + 1) * SF;
        float FA[C], bA[C], FBn[C], b3n[C], rc[C], mc[C], bb[3 * C];
        rag_tvdb_row<EX, C, D>(g, vA, b2c, dt, seam, FA, bA);
        if (g.real)
            for (int m = 0; m < C; m++)
                fax[w * SF + i0 + m] = FA[m];
        cp_async_wait<1>();
        landed(k + 1);
        __syncthreads();  // plane k+1 is staged, the A rows' EMFs of plane k are in
        const int s = slot(k + 1);
        u_read(s, w + 1, rc, mc);
        b_read(s, bb);
        {
            float vB[C][1], b3[C], rl[C], ml[C];
            face(rB, mB, rc, mc, vB);
#pragma unroll
            for (int m = 0; m < C; m++)
                b3[m] = bb[3 * m + 2];
            u_read(s, w, rl, ml);
            face(rl, ml, rc, mc, vA);
            rag_tvdb_row<EX, C, D>(g, vB, b3, dt, seam, FBn, b3n);
        }
        if (k + 1 == k1)
            before_next();
        if (owner) {
            float fa1[C];
            rag_lds<C, C>(fax + (w + 1) * SF + i0, fa1);
            const size_t cell0 = ((size_t)k * ny + j0 + w) * n + i0;
            float out[3 * C];
#pragma unroll
            for (int m = 0; m < C; m++) {
                float x = b1c[m];
                if (b1s != ub && m < own)
                    x = b1s[(cell0 + m) * 3];
                x = x - FA[m];
                x = x + fa1[m];
                x = x - FBc[m];
                x = x + FBn[m];
                out[3 * m] = x;
                out[3 * m + 1] = bA[m];
                out[3 * m + 2] = b3c[m];
            }
            if (C == 4 && pb == 16 && own == C) {
                stg_chunk<float, 3 * C>(bo + cell0 * 3, out);
            } else {
#pragma unroll
                for (int m = 0; m < C; m++)
                    if (m < own) {
                        bo[(cell0 + m) * 3] = out[3 * m];
                        bo[(cell0 + m) * 3 + 1] = out[3 * m + 1];
                        bo[(cell0 + m) * 3 + 2] = out[3 * m + 2];
                    }
            }
        }
#pragma unroll
        for (int m = 0; m < C; m++) {
            b1c[m] = bb[3 * m];
            b2c[m] = bb[3 * m + 1];
            rB[m] = rc[m];
            mB[m] = mc[m];
            FBc[m] = FBn[m];
            b3c[m] = b3n[m];
        }
        if (k + 1 < k1) {
            expect(k + 3);
            fence_proxy_async_smem();
            __syncthreads();  // plane k+1's slot has been read
            issue(k + 3);
        }
    }
    cp_async_wait<0>();
}

// ------------------------------------------------------------- launches

template <bool EX, int C, int D>
static cudaError_t launch_fx_rag(const FluidxArgs& a, const RagShape& sh, int pb, cudaStream_t s)
{
    static bool attr = false;
    const cudaError_t e = allow_smem(k_fluidx_rag<EX, C, D>, attr);
    if (e != cudaSuccess)
        return e;
    const dim3 grid((a.ny + a.P - 1) / a.P, a.nz, a.bs.count);
    return launch_after(k_fluidx_rag<EX, C, D>, grid, a.P * sh.G, rag_fluidx_smem(sh), s, a, sh, pb);
}

template <bool EX, int C, int D>
static cudaError_t launch_ad_rag(const AdvectArgs& a, const RagShape& sh, int pb, bool wu, cudaStream_t s)
{
    static bool attr[2] = {false, false};
    const cudaError_t e = wu ? allow_smem(k_advect_rag<EX, C, D, true>, attr[1])
                             : allow_smem(k_advect_rag<EX, C, D, false>, attr[0]);
    if (e != cudaSuccess)
        return e;
    const dim3 grid((a.ny + a.P - 1) / a.P, (a.nz + a.K - 1) / a.K, a.bs.count);
    const int nt = ((a.P + 1) * sh.G + 31) / 32 * 32;  // whole warps: groups past the halo pencil's repeat it
    const size_t smem = rag_advect_smem(sh, a.P);
    return launch_after(wu ? k_advect_rag<EX, C, D, true> : k_advect_rag<EX, C, D, false>, grid, nt, smem, s, a,
        sh, pb);
}

template <bool EX>
static cudaError_t fluidx_rag_set(const FluidxArgs& a, const RagShape& sh, int pb, cudaStream_t s)
{
    switch (sh.C * 10 + sh.T * sh.C - a.nx) {
    case 30: return launch_fx_rag<EX, 3, 0>(a, sh, pb, s);
    case 31: return launch_fx_rag<EX, 3, 1>(a, sh, pb, s);
    case 32: return launch_fx_rag<EX, 3, 2>(a, sh, pb, s);
    case 40: return launch_fx_rag<EX, 4, 0>(a, sh, pb, s);
    case 41: return launch_fx_rag<EX, 4, 1>(a, sh, pb, s);
    case 42: return launch_fx_rag<EX, 4, 2>(a, sh, pb, s);
    case 43: return launch_fx_rag<EX, 4, 3>(a, sh, pb, s);
    case 50: return launch_fx_rag<EX, 5, 0>(a, sh, pb, s);
    case 51: return launch_fx_rag<EX, 5, 1>(a, sh, pb, s);
    case 52: return launch_fx_rag<EX, 5, 2>(a, sh, pb, s);
    case 53: return launch_fx_rag<EX, 5, 3>(a, sh, pb, s);
    case 54: return launch_fx_rag<EX, 5, 4>(a, sh, pb, s);
    }
    return cudaErrorInvalidValue;
}

template <bool EX>
static cudaError_t advect_rag_set(const AdvectArgs& a, const RagShape& sh, int pb, bool wu, cudaStream_t s)
{
    switch (sh.C * 10 + sh.T * sh.C - a.nx) {
    case 30: return launch_ad_rag<EX, 3, 0>(a, sh, pb, wu, s);
    case 31: return launch_ad_rag<EX, 3, 1>(a, sh, pb, wu, s);
    case 32: return launch_ad_rag<EX, 3, 2>(a, sh, pb, wu, s);  // n = 1 only
    case 40: return launch_ad_rag<EX, 4, 0>(a, sh, pb, wu, s);
    case 41: return launch_ad_rag<EX, 4, 1>(a, sh, pb, wu, s);
    case 42: return launch_ad_rag<EX, 4, 2>(a, sh, pb, wu, s);
    case 50: return launch_ad_rag<EX, 5, 0>(a, sh, pb, wu, s);
    case 51: return launch_ad_rag<EX, 5, 1>(a, sh, pb, wu, s);
    case 52: return launch_ad_rag<EX, 5, 2>(a, sh, pb, wu, s);
    case 53: return launch_ad_rag<EX, 5, 3>(a, sh, pb, wu, s);
    }
    return cudaErrorInvalidValue;
}

}  // namespace mhd
