// FP32 kernels with FMA contraction (the production path).
#define MHD_SET_NAME set_f32_fast
#define MHD_REAL float
#define MHD_EXACT false
#include "kernels_impl.cuh"

namespace mhd {

const KernelSet* kernels_f32_fast() { return &set_f32_fast::kSet; }

static int pick_pencils(int nx, int ny, int target)
{
    int best = 1;
    for (int p = 1; p <= ny; p++)
        if (ny % p == 0 && (long long)p * nx <= target)
            best = p;
    return best;
}

int fluidx_pencils(int nx, int ny) { return pick_pencils(nx, ny, nx >= 256 ? nx : 256); }
int advect_pencils(int nx, int ny) { return pick_pencils(nx, ny, nx >= 256 ? nx : 256); }

cudaError_t launch_copy(const void* src, void* dst, size_t bytes, cudaStream_t s)
{
    if (bytes == 0)
        return cudaSuccess;
    const bool al16 = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
    if (al16 && bytes % 16 == 0) {
        size_t n16 = bytes / 16;
        int blocks = (int)((n16 + 255) / 256);
        if (blocks > 152 * 16)
            blocks = 152 * 16;
        return launch_after(k_copy16, blocks, 256, 0, s, static_cast<const uint4*>(src), static_cast<uint4*>(dst), n16);
    } else {
        size_t n4 = bytes / 4;
        int blocks = (int)((n4 + 255) / 256);
        if (blocks > 152 * 16)
            blocks = 152 * 16;
        return launch_after(k_copy4, blocks, 256, 0, s, static_cast<const float*>(src), static_cast<float*>(dst), n4);
    }
}

int launch_copy2(const void* src0, void* dst0, size_t bytes0, const void* src1, void* dst1, size_t bytes1,
                 cudaStream_t s, cudaError_t* e)
{
    const uintptr_t al = reinterpret_cast<uintptr_t>(src0) | reinterpret_cast<uintptr_t>(dst0) |
                         reinterpret_cast<uintptr_t>(src1) | reinterpret_cast<uintptr_t>(dst1);
    if ((al & 15) != 0 || bytes0 % 16 != 0 || bytes1 % 16 != 0 || bytes0 == 0 || bytes1 == 0) {
        *e = launch_copy(src0, dst0, bytes0, s);
        if (*e == cudaSuccess)
            *e = launch_copy(src1, dst1, bytes1, s);
        return 2;
    }
    const size_t n0 = bytes0 / 16, n1 = bytes1 / 16, b = (n0 + n1 + 255) / 256;
    *e = launch_after(k_copy16x2, (unsigned)(b < 152 * 16 ? b : 152 * 16), 256, 0, s, static_cast<const uint4*>(src0),
                      static_cast<uint4*>(dst0), n0, static_cast<const uint4*>(src1), static_cast<uint4*>(dst1), n1);
    return 1;
}

}  // namespace mhd
