// Ragged-pencil kernels, FAST policy (see mhd_ragged.cuh), and their launch rules
#include "mhd_ragged.cuh"

namespace mhd {

cudaError_t fluidx_rag_fast(const FluidxArgs& a, const RagShape& sh, int pb, cudaStream_t s)
{
    return fluidx_rag_set<false>(a, sh, pb, s);
}

cudaError_t advect_rag_fast(const AdvectArgs& a, const RagShape& sh, int pb, bool wu, cudaStream_t s)
{
    return advect_rag_set<false>(a, sh, pb, wu, s);
}

// The C of 3, 4, 5 with the fewest lane slots G C (4 first on a tie: its
// shared-memory accesses are 16 bytes wide).  `ahead`: the cells after a thread's
// own that an exchange asks for (fluidx 1, tvdb 2): the last thread's come from
// cells C-L .. C-L+ahead-1 of thread 0, so L >= ahead.  C = 0 if there is none
// (ahead 2 and n - 1 a multiple of 60).
RagShape rag_shape(int n, int ahead)
{
    RagShape best{0, 0, 0};
    const int order[3] = {4, 5, 3};
    for (int q = 0; q < 3; q++) {
        const int C = order[q], T = (n + C - 1) / C;
        if (n - (T - 1) * C < ahead && n > 1)
            continue;
        const int G = (T <= 8) ? 8 : (T <= 16 ? 16 : (T + 31) / 32 * 32);
        if (!best.C || G * C < best.G * best.C)
            best = RagShape{C, T, G};
    }
    return best;
}

int rag_fluidx_parts(int nx, int ny, int nz)
{
    const int P = rag_pencils(rag_shape(nx, 1));
    return (ny + P - 1) / P * nz;
}

cudaError_t fluidx_rag_exact(const FluidxArgs& a, const RagShape& sh, int pb, cudaStream_t s);
cudaError_t advect_rag_exact(const AdvectArgs& a, const RagShape& sh, int pb, bool wu, cudaStream_t s);

// the largest piece that every pencil of n cells starts on and consists of
static int rag_piece(int n, uintptr_t al)
{
    return (n % 4 == 0 && (al & 15) == 0) ? 16 : (n % 2 == 0 && (al & 7) == 0 ? 8 : 4);
}

cudaError_t fluidx_ragged(const FluidxArgs& in, bool exact, cudaStream_t s)
{
    FluidxArgs a = in;
    const RagShape sh = rag_shape(a.nx, 1);
    const uintptr_t al = reinterpret_cast<uintptr_t>(a.u_out) | reinterpret_cast<uintptr_t>(a.uu) |
                         reinterpret_cast<uintptr_t>(a.ub) | (a.bs.count > 1 ? a.bs.u | a.bs.b : 0);
    const int pb = rag_piece(a.nx, al);
    a.P = rag_pencils(sh);
    if (a.P * sh.G > kRagThreads)
        return cudaErrorInvalidValue;
    return exact ? fluidx_rag_exact(a, sh, pb, s) : fluidx_rag_fast(a, sh, pb, s);
}

// J pencils per CTA: five groups of 32 lanes or ten of 16 (the group of the
// halo pencil is the price of a small J).  K planes: the K with the least waves of
// CTAs x (K + 1.5), as a6_planes (four
// steps of 100 x 72 x 72: 0.95 ms, 1.05 with the most planes that left 608 CTAs).
cudaError_t advect_ragged(const AdvectArgs& in, bool exact, cudaStream_t s)
{
    AdvectArgs a = in;
    const RagShape sh = rag_shape(a.nx, 2);
    const bool wu = a.w != nullptr && (reinterpret_cast<uintptr_t>(a.w) & 7) == 0;
    const uintptr_t al = reinterpret_cast<uintptr_t>(a.b_out) | reinterpret_cast<uintptr_t>(a.ub) |
                         (wu ? reinterpret_cast<uintptr_t>(a.w) : 0) |
                         (a.bs.count > 1 ? a.bs.b | (wu ? a.bs.w : 0) : 0);
    const int pb = rag_piece(a.nx, al);
    const int jt = tune_value(TUNE_ADVECT_J), kt = tune_value(TUNE_ADVECT_K);
    int jmax = (sh.G > 128) ? 1 : (sh.G >= 64 ? 2 : 160 / sh.G - 1);  // at most 512 threads
    if (jt > 0 && (jt + 1) * sh.G <= 512)
        jmax = jt;
    const int nj = (a.ny + jmax - 1) / jmax;
    a.P = (a.ny + nj - 1) / nj;
    const int nt = ((a.P + 1) * sh.G + 31) / 32 * 32;
    const long long wave = 152LL * (65536 / (nt * 112) > 0 ? 65536 / (nt * 112) : 1);  // at 97-120 registers
    long long best = -1;
    for (int k = 1; k <= 32 && k <= a.nz; k++) {
        const long long cost = ((long long)nj * ((a.nz + k - 1) / k) * a.bs.count + wave - 1) / wave * (2 * k + 3);
        if (kt ? (k == 1 || k == kt) : (best < 0 || cost < best)) {
            best = cost;
            a.K = k;
        }
    }
    return exact ? advect_rag_exact(a, sh, pb, wu, s) : advect_rag_fast(a, sh, pb, wu, s);
}

}  // namespace mhd
