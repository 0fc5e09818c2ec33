// k_render.cu -- frame rasteriser: the reference's CPU animator frame
// (sim/animator.go:55-103 CurrentFrame) as two CUDA kernels writing a headless
// NRGBA buffer instead of an OpenGL window.
//
// The reference sorts particles by -Z (sim/heap.go:229-268 QuickSort) and
// paints a disk of radius 4 pixels for each in that order
// (gx/graphics.go:90-107 DrawDisk), coloured by ParaRamp
// (gx/graphics.go:156-164) of min(rho / (m N 10) * 256, 255). Painting in order
// means every pixel shows the LAST disk that covers it, so here each particle
// raises the pixels it covers to its draw rank with atomicMax (k_draw), and a
// second pass colours each pixel from the winning particle's density
// (k_resolve). Pixel tests keep the reference's FP32 arithmetic and rounding
// (no contraction), so frames are identical to a sequential painter.
#include "physics.cuh"

namespace sphgpu {

__constant__ uchar4 c_ramp[256];

#define GRID_STRIDE(i, n) \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

// A warp draws eight disks, one after the other, three pixel rows of ten lanes
// each at a time (a disk's box has at most ten by ten pixels), so that a row's
// pixels leave in one or two sectors; bound by the L2's reductions. With a
// thread per disk the 50 pixels of each were a sector apiece: 29 us for
// 100,000 disks on 1280 x 720, this form 15.
constexpr int kDisksPerWarp = 8;

__global__ void __launch_bounds__(128) k_draw(Ctx c, PArrays A, const int32_t *zrank, int32_t *rslot, int32_t *fb, int W, int H) {
    const int lane = threadIdx.x & 31, col = lane % 10, row = lane / 10;
    const int64_t i0 = (blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * kDisksPerWarp, i = i0 + lane;
    if (i0 >= c.n) return;
    const float rad = 4.f;
    float cx = 0.f, cy = 0.f;
    int r = 0, xa = 0, xb = -1, ya = 0, yb = -1;
    if (lane < kDisksPerWarp && i < c.n) {
        const int32_t id = A.id[i];
        r = zrank ? zrank[id] : id;  // default: caller order, the last on top
        rslot[r] = (int32_t)i;
        const double2 p = A.pos[i];
        // x := float32(Pos.X) * float32(W)
        cx = __fmul_rn(emu_d2f(p.x), (float)W);
        cy = __fmul_rn(emu_d2f(p.y), (float)H);
        const float fxa = floorf(__fsub_rn(cx, rad)), fxb = ceilf(__fadd_rn(cx, rad));
        const float fya = floorf(__fsub_rn(cy, rad)), fyb = ceilf(__fadd_rn(cy, rad));
        // pixels outside the canvas are ignored (image.NRGBA.Set); NaN positions draw nothing
        if (fxb >= 0.f && fxa <= (float)(W - 1) && fyb >= 0.f && fya <= (float)(H - 1)) {
            xa = max((int)fxa, 0);
            xb = min((int)fxb, W - 1);
            ya = max((int)fya, 0);
            yb = min((int)fyb, H - 1);
        }
    }
#pragma unroll
    for (int d = 0; d < kDisksPerWarp; d++) {
        const float dcx = __shfl_sync(0xffffffffu, cx, d), dcy = __shfl_sync(0xffffffffu, cy, d);
        const int dxb = __shfl_sync(0xffffffffu, xb, d), dyb = __shfl_sync(0xffffffffu, yb, d);
        const int rank = __shfl_sync(0xffffffffu, r, d);
        const int x = __shfl_sync(0xffffffffu, xa, d) + col;
        const float dx = __fsub_rn((float)x, dcx);
        const float dx2 = __fmul_rn(dx, dx);
        const bool in = row < 3 && x <= dxb;
        for (int y = __shfl_sync(0xffffffffu, ya, d) + row; y <= dyb; y += 3) {
            const float dy = __fsub_rn((float)y, dcy);
            if (in && __fadd_rn(dx2, __fmul_rn(dy, dy)) <= __fmul_rn(rad, rad)) atomicMax(&fb[(int64_t)y * W + x], rank);
        }
    }
}

// uint8(math.Min(v, 255)): truncation; negative and NaN give 0
__device__ __forceinline__ int colour_index(double v) {
    const uint32_t h = emu_hi(v);
    if (h >= 0x40700000u) return h <= 0x7ff00000u && !(h == 0x7ff00000u && emu_lo(v)) ? 255 : 0;  // 256 and above; NaN, negative
    return h < 0x3ff00000u ? 0 : (int)(((h & 0xfffffu) | 0x100000u) >> (1043u - (h >> 20)));
}

// The quotient on the integer pipes: the FP64 unit was 82 % busy with divisions
// (1280 x 720: 26 us, now 10).
__global__ void k_resolve(const int32_t *fb, const int32_t *rslot, const double *rho, int64_t n_eval, double den,
                          uchar4 *out, int64_t npix) {
    const EmuDivisor D = emu_divisor(den);
    GRID_STRIDE(p, npix) {
        const int32_t r = fb[p];
        uchar4 col = make_uchar4(0, 0, 0, 255);  // gx.BLACK
        if (r >= 0) {
            const int32_t s = rslot[r];
            const double rh = s < n_eval ? rho[s] : 0.0;
            // float64(Rho / (m * float64(N*10)) * 256), then uint8(math.Min(., 255))
            col = c_ramp[colour_index(emu_mul(emu_div(rh, D, den), 256.0))];
        }
        out[p] = col;
    }
}

int set_ramp(const unsigned char rgba[256 * 4]) {
    return cudaMemcpyToSymbol(c_ramp, rgba, 256 * 4) == cudaSuccess ? 0 : -1;
}

void launch_render(const Ctx &c, const Launch &L, const PArrays &A, const int32_t *zrank, int32_t *rslot,
                   int32_t *fb, const double *rho, int64_t n_eval, double mass, int W, int H, uchar4 *out) {
    const int64_t npix = (int64_t)W * H;
    cudaMemsetAsync(fb, 0xff, npix * sizeof(int32_t), L.stream);  // -1: no disk
    const int64_t per_block = 4 * kDisksPerWarp;
    k_draw<<<(int)((c.n + per_block - 1) / per_block), 128, 0, L.stream>>>(c, A, zrank, rslot, fb, W, H);
    const int64_t rg = std::min<int64_t>((npix + 255) / 256, (int64_t)L.sms * 16);
    k_resolve<<<(int)std::max<int64_t>(rg, 1), 256, 0, L.stream>>>(fb, rslot, rho, n_eval, mass * (double)(c.n * 10), out, npix);
}

}  // namespace sphgpu
