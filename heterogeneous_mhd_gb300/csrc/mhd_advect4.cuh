// advectbyzx walking along x (C/advectbyzx.c:14-23 with A1 C/advectbyzxA1.c:18-63,
// A2 C/advectbyzxA2.c:9-28, B1 C/advectbyzxB1.c:19-62, B2 C/advectbyzxB2.c:9-28
// and tvdb C/tvdb.c:10-91), for the x sweep of the transposed state.
//
// Every thread owns two whole tvdb rows: an A row (b(2) advected with the
// face velocity of pencils j-1, j) and a B row (b(3) with pencils k-1, k).
// It walks its rows along x in chunks of four cells and carries the stencil
// in registers: on reading position p it forms vx(p), the smoothed vg(p-1),
// the half step at p-2 and the limited flux at p-4, so no value moves between
// threads while a row is computed (no shuffles, no barriers in the stencil).
//
// A CTA covers a tile of 32 pencils along j (the lanes) by KT planes along k
// (the warps).  Warp w < KT owns the A and B rows of pencil (j0+lane, k0+w);
// warp KT owns the B rows of plane k0+KT and, in lanes 0..KT-1, the A rows of
// pencil (j0+32, k0+lane).  Per chunk the EMFs of the neighbouring rows meet
// (FB of plane k+1 through shared memory, FA of pencil j+1 by a shuffle, from
// warp KT for lane 31) and warp w < KT applies the float updates in the order
// of A1, A2, B1, B2:
//   b1_out = (((b1 - FA(j,k)) + FA(j+1,k)) - FB(j,k)) + FB(j,k+1).
//
// Input chunks (u pencils j0-1..j0+32 x k0-1..k0+KT and b pencils
// j0..j0+32 x k0..k0+KT, four cells each, in their global layout: 80-byte u
// and 48-byte b records, which consecutive lanes read with 16-byte loads
// without bank conflicts) arrive by cp.async in a ring of NS buffers.  The
// CTAs are persistent: each takes an equal share of the (tile, chunk) work of
// its box (whole tiles, then x segments of the tiles left over), so no CTA
// waits in a partial last wave; a segment starts one chunk early and ends one
// chunk late (the stencil's reach, 4 cells each way, is one chunk).
#pragma once
#include <type_traits>

#include "mhd_advect2.cuh"
#include "mhd_ptx.cuh"

namespace mhd {

constexpr int kA4X = 4;                  // cells per chunk
constexpr int kA4J = 32;                 // pencils per tile along j
constexpr int kA4UC = kA4J + 2;          // staged u columns j0-1..j0+32
constexpr int kA4BC = kA4J + 1;          // staged b columns j0..j0+32
constexpr int kA4BR = kA4BC * 3 * kA4X;  // floats of one staged b plane

__host__ __device__ inline int advect4_threads(int KT) { return (KT + 1) * 32; }

// ring of NS (u, b) chunk buffers, then the EMF exchange: FB [KT+1][32] and
// FA [KT] float4
// staged u record of 4 cells in floats: the u records (20), or the (rho, m_x)
// side array's (8, padded to 12 so that consecutive lanes read them with
// 16-byte loads without bank conflicts)
__host__ __device__ constexpr int advect4_urec(bool wu) { return wu ? 12 : 5 * kA4X; }

__host__ __device__ inline size_t advect4_smem_bytes(int KT, int NS, bool wu = false)
{
    const size_t buf = (size_t)(KT + 2) * kA4UC * advect4_urec(wu) + (size_t)(KT + 1) * kA4BR;
    return (NS * buf + 4 * ((size_t)(KT + 1) * 32 + KT)) * sizeof(float);
}

// One tvdb row walked along x.  B is the first cell of the chunk being read;
// the state holds what the stencil still needs from the cells before it.
template <bool EX>
struct XRow {
    float vx2, vx1;        // vx(B-2), vx(B-1)
    float bv[kA4X];        // b(B-4) .. b(B-1)
    float vg2, t22, f13;   // vg(B-2), t2(B-2), f1(B-3)
    float vb5, vb4, vb3;   // vb(B-5), vb(B-4), vb(B-3)
    float vh4, vh3;        // vh(B-4), vh(B-3)
    float fl5;             // flux(B-5)

    __device__ __forceinline__ void reset()
    {
        vx2 = vx1 = vg2 = t22 = f13 = vb5 = vb4 = vb3 = vh4 = vh3 = fl5 = 0.f;
#pragma unroll
        for (int m = 0; m < kA4X; m++)
            bv[m] = 0.f;
    }

    // vx, b of cells B..B+3 in; F = flux(i-1) and the advected b of cells
    // i = B-4..B-1 out (the same per-cell expressions as tvdb_row).
    __device__ __forceinline__ void step(const float (&vx)[kA4X], const float (&bc)[kA4X], float dt,
                                         float (&F)[kA4X], float (&bn)[kA4X])
    {
        float VG[4], T2[4], VH[4], F1[4], VB[4], FL[4];
        // vg(B+m-1)
        VG[0] = tvdb_smooth<float, EX>(vx2, vx1, vx[0]);
        VG[1] = tvdb_smooth<float, EX>(vx1, vx[0], vx[1]);
        VG[2] = tvdb_smooth<float, EX>(vx[0], vx[1], vx[2]);
        VG[3] = tvdb_smooth<float, EX>(vx[1], vx[2], vx[3]);
        // t2(B+m-1) = b vg
        T2[0] = tvdb_prod<float, EX>(bv[3], VG[0]);
#pragma unroll
        for (int m = 1; m < 4; m++)
            T2[m] = tvdb_prod<float, EX>(bc[m - 1], VG[m]);
        // vh(B+m-2) and the upwind f1(B+m-2)
        VH[0] = tvdb_vh<float, EX>(vg2, VG[0]);
        F1[0] = (VH[0] > 0.f) ? t22 : T2[0];
#pragma unroll
        for (int m = 1; m < 4; m++) {
            VH[m] = tvdb_vh<float, EX>(VG[m - 1], VG[m]);
            F1[m] = (VH[m] > 0.f) ? T2[m - 1] : T2[m];
        }
        // half step b1(B+m-2), vb = vg b1
        VB[0] = tvdb_prod<float, EX>(vg2, tvdb_half<float, EX>(bv[2], F1[0], f13, dt));
        VB[1] = tvdb_prod<float, EX>(VG[0], tvdb_half<float, EX>(bv[3], F1[1], F1[0], dt));
        VB[2] = tvdb_prod<float, EX>(VG[1], tvdb_half<float, EX>(bc[0], F1[2], F1[1], dt));
        VB[3] = tvdb_prod<float, EX>(VG[2], tvdb_half<float, EX>(bc[1], F1[3], F1[2], dt));
        // flux(B+m-4) from vb(B+m-5 .. B+m-2) and vh(B+m-4)
        FL[0] = tvdb_flux<float, EX>(vb5, vb4, vb3, VB[0], vh4, dt);
        FL[1] = tvdb_flux<float, EX>(vb4, vb3, VB[0], VB[1], vh3, dt);
        FL[2] = tvdb_flux<float, EX>(vb3, VB[0], VB[1], VB[2], VH[0], dt);
        FL[3] = tvdb_flux<float, EX>(VB[0], VB[1], VB[2], VB[3], VH[1], dt);
        // F(i) = flux(i-1), b - (flux - flux(i-1))
        F[0] = fl5;
#pragma unroll
        for (int m = 1; m < 4; m++)
            F[m] = FL[m - 1];
#pragma unroll
        for (int m = 0; m < 4; m++)
            bn[m] = tvdb_new<float, EX>(bv[m], FL[m], F[m]);
        // advance by one chunk
        vx2 = vx[2];
        vx1 = vx[3];
#pragma unroll
        for (int m = 0; m < 4; m++)
            bv[m] = bc[m];
        vg2 = VG[3];
        t22 = T2[3];
        f13 = F1[3];
        vb5 = VB[1];
        vb4 = VB[2];
        vb3 = VB[3];
        vh4 = VH[2];
        vh3 = VH[3];
        fl5 = FL[3];
    }
};

// rho and m_x (components 0, 1) of the four cells of a staged u record, or of
// a side-array record (rho0, mx0, rho1, mx1, rho2, mx2, rho3, mx3)
template <bool WU>
__device__ __forceinline__ void a4_rho_mx(const float* p, float (&rho)[4], float (&mx)[4])
{
    const float4* q = reinterpret_cast<const float4*>(p);
    if constexpr (WU) {
        const float4 v0 = q[0], v1 = q[1];
        rho[0] = v0.x, mx[0] = v0.y;
        rho[1] = v0.z, mx[1] = v0.w;
        rho[2] = v1.x, mx[2] = v1.y;
        rho[3] = v1.z, mx[3] = v1.w;
    } else {
        const float4 v0 = q[0], v1 = q[1], v2 = q[2], v3 = q[3], v4 = q[4];
        rho[0] = v0.x, mx[0] = v0.y;
        rho[1] = v1.y, mx[1] = v1.z;
        rho[2] = v2.z, mx[2] = v2.w;
        rho[3] = v3.w, mx[3] = v4.x;
    }
}

__device__ __forceinline__ void a4_b(const float* p, float (&b)[12])
{
    const float4* q = reinterpret_cast<const float4*>(p);
#pragma unroll
    for (int v = 0; v < 3; v++) {
        const float4 x = q[v];
        b[4 * v] = x.x, b[4 * v + 1] = x.y, b[4 * v + 2] = x.z, b[4 * v + 3] = x.w;
    }
}

// raw face velocity (C/advectbyzxA1.c:34, C/advectbyzxB1.c:34): pencil below (m) and current (c)
template <bool EX>
__device__ __forceinline__ void a4_face(const float (&rm)[4], const float (&mm)[4], const float (&rc)[4],
                                        const float (&mc)[4], float (&vx)[4])
{
#pragma unroll
    for (int m = 0; m < 4; m++)
        vx[m] = tvdb_face<float, EX>(mm[m], mc[m], rm[m], rc[m]);
}

// CTAs per SM the register budget is sized for (shared memory allows as many,
// except KT = 2 with three buffers: 4)
__host__ __device__ constexpr int advect4_min_ctas(int KT, int NS)
{
    return KT == 2 ? 5 : (KT == 4 ? 3 : 1);
}

// WU: the u chunks come from the (rho, m_x) side array a.w (8 bytes per cell)
template <bool EX, int KT, int NS, bool WU = false>
__global__ void __launch_bounds__((KT + 1) * 32, advect4_min_ctas(KT, NS)) k_advect4(AdvectArgs a)
{
    after_previous();
    static_assert(NS == 2 || NS == 3, "two or three chunk buffers");
    select_box(a, blockIdx.z);
    constexpr int NW = KT + 1;                            // warps
    constexpr int REC = advect4_urec(WU), UR = kA4UC * REC;  // staged u record and plane (floats)
    constexpr int UCELL = WU ? 2 : 5, PPR = WU ? 2 : 5;      // source floats per cell, 16-byte pieces per record
    constexpr int UBUF = (KT + 2) * UR, BBUF = (KT + 1) * kA4BR;
    constexpr int UP = kA4UC * PPR, BP = kA4BC * 3;          // 16-byte pieces of a staged plane
    constexpr int UQ = (UP + 31) / 32, BQ = (BP + 31) / 32;
    extern __shared__ __align__(16) float a4_smem[];
    float* Us = a4_smem;                                  // [NS][KT+2][34][REC]
    float* Bs = Us + NS * UBUF;                           // [NS][KT+1][33][12]
    float4* FBx = reinterpret_cast<float4*>(Bs + NS * BBUF);  // [KT+1][32]
    float4* FAx = FBx + NW * 32;                              // [KT]

    const int nx = a.nx, ny = a.ny, nz = a.nz;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool bw = (w == KT);
    const float dt = load_dt<float>(a.dt_ptr, a.dt_val);
    const float* uu = static_cast<const float*>(a.uu);
    const float* ub = static_cast<const float*>(a.ub);
    const float* usrc = WU ? static_cast<const float*>(a.w) : uu;  // what the u chunks are staged from
    const float* b1s = static_cast<const float*>(a.b1_src);
    float* bo = static_cast<float*>(a.b_out);
    const bool b1_staged = (b1s == ub);

    // this thread's rows: A at tile (ja, ka), B at (jb, kb); their staged records
    const int ja = bw ? kA4J : lane, ka = bw ? (lane < KT ? lane : 0) : w;
    const int jb = lane, kb = bw ? KT : w;
    const int uAm = (ka + 1) * UR + ja * REC, uAc = (ka + 1) * UR + (ja + 1) * REC;
    const int uBm = kb * UR + (jb + 1) * REC, uBc = (kb + 1) * UR + (jb + 1) * REC;
    const int bA = ka * kA4BR + ja * 12, bB = kb * kA4BR + jb * 12;

    // Work: whole tiles in rounds (CTA i takes tiles i, i + P, ...: all CTAs
    // walk x together, so the halo pencils a tile shares with its neighbours
    // are read from L2 the second time), then the tiles left over, split in
    // x among all CTAs (tile-major, so concurrent segments stay close in x).
    const int NC = nx / kA4X, tj = ny / kA4J, tk = nz / KT;
    const int ntiles = tj * tk, P = (int)gridDim.x, full = ntiles / P;
    const long long rest = (long long)(ntiles - full * P) * NC;
    long long ws = rest * blockIdx.x / P;
    const long long wend = rest * (blockIdx.x + 1) / P;

    for (int round = 0;; round++) {
        int tile, c0, c1;
        if (round < full) {
            tile = (int)blockIdx.x + round * P;
            c0 = 0;
            c1 = NC;
        } else {
            if (ws >= wend)
                break;
            const long long u = ws / NC;
            c0 = (int)(ws - u * NC);
            c1 = (int)((wend - ws < (long long)(NC - c0)) ? (c0 + (wend - ws)) : NC);
            ws += c1 - c0;
            tile = full * P + (int)u;
        }
        const int j0 = (tile % tj) * kA4J, k0 = (tile / tj) * KT;

        // Staging: warp w copies staged u plane w (and warp 0 also plane KT+1)
        // and staged b plane w; lane l copies the 16-byte pieces l + 32 q of a
        // plane.  Offsets in floats of chunk 0: the k part per plane, the j and
        // component part per piece (-1: no piece).
        int ucol[UQ], bcol[BQ];
#pragma unroll
        for (int q = 0; q < UQ; q++) {
            const int p = lane + 32 * q, c = p / PPR, pc = p - PPR * c;
            int jg = j0 + c - 1;
            jg = (jg < 0) ? jg + ny : (jg >= ny ? jg - ny : jg);
            ucol[q] = (p < UP) ? jg * nx * UCELL + pc * 4 : -1;
        }
#pragma unroll
        for (int q = 0; q < BQ; q++) {
            const int p = lane + 32 * q, c = p / 3, pc = p - 3 * c;
            int jg = j0 + c;
            jg = (jg >= ny) ? jg - ny : jg;
            bcol[q] = (p < BP) ? jg * nx * 3 + pc * 4 : -1;
        }
        auto kwrap = [&](int k) { return (k < 0) ? k + nz : (k >= nz ? k - nz : k); };
        const int urow0 = kwrap(k0 + w - 1) * ny * nx * UCELL, urow1 = kwrap(k0 + KT) * ny * nx * UCELL;
        // shared offset of piece lane + 32 q of a staged plane: record p / PPR, piece p % PPR
        const int ulane = WU ? ((lane >> 1) * REC + (lane & 1) * 4) : lane * 4;
        constexpr int UQSTEP = WU ? 16 * REC : 128;
        const int brow = kwrap(k0 + w) * ny * nx * 3;
        // virtual chunk v (c0-1 .. c1, periodic) into ring buffer s
        auto load_chunk = [&](int v, int s) {
            const int xr = (v < 0) ? v + NC : (v >= NC ? v - NC : v);
            float* ud0 = Us + s * UBUF + w * UR + ulane;
            float* bd0 = Bs + s * BBUF + w * kA4BR + lane * 4;
            const float* us0 = usrc + urow0 + xr * (UCELL * kA4X);
#pragma unroll
            for (int q = 0; q < UQ; q++)
                if (ucol[q] >= 0)
                    cp_async16(ud0 + UQSTEP * q, us0 + ucol[q]);
            if (w == 0) {  // the last staged u plane (k0 + KT)
                float* ud1 = Us + s * UBUF + (KT + 1) * UR + ulane;
                const float* us1 = usrc + urow1 + xr * (UCELL * kA4X);
#pragma unroll
                for (int q = 0; q < UQ; q++)
                    if (ucol[q] >= 0)
                        cp_async16(ud1 + UQSTEP * q, us1 + ucol[q]);
            }
            const float* bs0 = ub + brow + xr * (3 * kA4X);
#pragma unroll
            for (int q = 0; q < BQ; q++)
                if (bcol[q] >= 0)
                    cp_async16(bd0 + 128 * q, bs0 + bcol[q]);
        };

        const int nv = c1 - c0 + 2;
        __syncthreads();  // the previous segment no longer reads the buffers
#pragma unroll
        for (int i = 0; i < NS - 1; i++) {
            if (i < nv)
                load_chunk(c0 - 1 + i, i);
            cp_async_commit();
        }
        XRow<EX> RA, RB;
        RA.reset();
        RB.reset();
        float bdp[4] = {0.f, 0.f, 0.f, 0.f};  // b(1) of the chunk before the one read
        // global cell of the first output cell of warp w's pencil (chunk c0)
        const size_t cell0 = ((size_t)(k0 + w) * ny + (j0 + lane)) * nx + (size_t)c0 * kA4X;
        // chunk i of the segment (virtual chunk c0-1+i) from ring buffer S
        auto chunk = [&](int i, auto sbuf) {
            constexpr int S = decltype(sbuf)::value;
            cp_async_wait<NS - 2>();
            __syncthreads();  // chunk i has landed everywhere; chunk i-1's buffer is free
            if (i + NS - 1 < nv)
                load_chunk(c0 - 1 + i + NS - 1, (S + NS - 1) % NS);
            cp_async_commit();
            const float* U = Us + S * UBUF;
            const float* Bv = Bs + S * BBUF;
            float vxA[4], vxB[4], bvA[4], bvB[4], bd1[4];
            {
                float rm[4], mm[4], rc[4], mc[4], rk[4], mk[4];
                a4_rho_mx<WU>(U + uAm, rm, mm);
                a4_rho_mx<WU>(U + uAc, rc, mc);
                a4_rho_mx<WU>(U + uBm, rk, mk);
                a4_face<EX>(rm, mm, rc, mc, vxA);
                float ba[12];
                a4_b(Bv + bA, ba);
                if (!bw) {  // the A and B rows of one pencil share its u and b records
                    a4_face<EX>(rk, mk, rc, mc, vxB);
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        bvA[m] = ba[3 * m + 1];
                        bvB[m] = ba[3 * m + 2];
                        bd1[m] = ba[3 * m];
                    }
                } else {
                    float rb[4], mb[4], bb[12];
                    a4_rho_mx<WU>(U + uBc, rb, mb);
                    a4_face<EX>(rk, mk, rb, mb, vxB);
                    a4_b(Bv + bB, bb);
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        bvA[m] = ba[3 * m + 1];
                        bvB[m] = bb[3 * m + 2];
                        bd1[m] = 0.f;
                    }
                }
            }
            float FA[4], BNA[4], FB[4], BNB[4];
            RA.step(vxA, bvA, dt, FA, BNA);
            RB.step(vxB, bvB, dt, FB, BNB);
            if (i >= 2) {  // the chunk before the one read (c0 + i - 2) is complete
                FBx[w * 32 + lane] = make_float4(FB[0], FB[1], FB[2], FB[3]);
                if (bw && lane < KT)
                    FAx[lane] = make_float4(FA[0], FA[1], FA[2], FA[3]);
                __syncthreads();
                if (!bw) {
                    float fan[4];
#pragma unroll
                    for (int m = 0; m < 4; m++)
                        fan[m] = __shfl_down_sync(kFull, FA[m], 1);
                    if (lane == 31) {
                        const float4 t = FAx[w];
                        fan[0] = t.x, fan[1] = t.y, fan[2] = t.z, fan[3] = t.w;
                    }
                    const float4 fbn = FBx[(w + 1) * 32 + lane];
                    const float fbv[4] = {fbn.x, fbn.y, fbn.z, fbn.w};
                    const size_t cell = cell0 + (size_t)(i - 2) * kA4X;
                    float b1v[4];
                    if (b1_staged) {
#pragma unroll
                        for (int m = 0; m < 4; m++)
                            b1v[m] = bdp[m];
                    } else {
#pragma unroll
                        for (int m = 0; m < 4; m++)
                            b1v[m] = b1s[(cell + m) * 3];
                    }
                    float out[12];
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        float x = b1v[m];
                        x = x - FA[m];
                        x = x + fan[m];
                        x = x - FB[m];
                        x = x + fbv[m];
                        out[3 * m] = x;
                        out[3 * m + 1] = BNA[m];
                        out[3 * m + 2] = BNB[m];
                    }
                    stg_chunk<float, 12>(bo + cell * 3, out);
                }
            }
#pragma unroll
            for (int m = 0; m < 4; m++)
                bdp[m] = bd1[m];
        };
        // unrolled by the ring depth: every buffer offset is a constant
        using S0 = std::integral_constant<int, 0>;
        using S1 = std::integral_constant<int, 1>;
        using S2 = std::integral_constant<int, (NS > 2 ? 2 : 0)>;
        int i = 0;
        for (; i + NS <= nv; i += NS) {
            chunk(i, S0{});
            chunk(i + 1, S1{});
            if constexpr (NS == 3)
                chunk(i + 2, S2{});
        }
        if (i < nv)
            chunk(i, S0{});
        if (NS == 3 && i + 1 < nv)
            chunk(i + 1, S1{});
    }
    cp_async_wait<0>();
}

}  // namespace mhd
