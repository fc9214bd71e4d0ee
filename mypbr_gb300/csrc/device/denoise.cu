// The denoiser of the reference (include/denoiser.h:45-193) on the device:
// firefly clamp, then edge-avoiding a-trous iterations with the SVGF
// variance-guided luminance weight, on lighting = radiance / (albedo + 1e-3).
//
// Iteration i spreads its 5 x 5 B3-spline taps 2^i pixels apart, so the taps
// of pixel (x, y) all lie on the lattice {(x + a s, y + b s)} of spacing s.
// A block takes one phase (x mod s, y mod s) of the image and a 16 x 16 tile
// of that phase's lattice: it stages the 20 x 20 lattice points the tile's
// taps reach (lighting + variance, albedo, normal: 48 B each) in shared
// memory once, and every staged point then serves up to 25 outputs. The
// variance blur (3 x 3 at step 1, denoiser.h:158-178) is a separate pass.
// Arithmetic is FP32; the frame comes in and goes out in FP64.
#include <algorithm>
#include <string>

#include "dev_math.cuh"
#include "gpu_scene.h"

namespace mypbr_dev {
namespace {

constexpr int kTile = 16;
constexpr int kHalo = 2;
constexpr int kSpan = kTile + 2 * kHalo;

MYPBR_DEV float lum(float4 c) { return dot_x(f3(0.2126f, 0.7152f, 0.0722f), f3(c)); }

// lighting = radiance / (albedo + eps), its variance over luminance(albedo + eps)^2
__global__ void k_dn_prepare(const double* rad, const double* alb, const double* nrm, const double* var, int n,
                             float4* L, float4* A, float4* N) {
    const float eps = 1e-3f;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        float a0 = float(alb[3 * k]), a1 = float(alb[3 * k + 1]), a2 = float(alb[3 * k + 2]);
        float e0 = a0 + eps, e1 = a1 + eps, e2 = a2 + eps;
        float la = 0.2126f * e0 + 0.7152f * e1 + 0.0722f * e2;
        L[k] = make_float4(float(rad[3 * k]) / e0, float(rad[3 * k + 1]) / e1, float(rad[3 * k + 2]) / e2,
                           float(var[k]) / (la * la));
        A[k] = make_float4(a0, a1, a2, 0.0f);
        N[k] = make_float4(float(nrm[3 * k]), float(nrm[3 * k + 1]), float(nrm[3 * k + 2]), 0.0f);
    }
}

// remove_fireflies (denoiser.h:90-111): a pixel brighter than its eight
// neighbours whose deviation exceeds half its luminance is scaled down to the
// brightest neighbour. Reads src, writes dst (every pixel).
__global__ void k_dn_fireflies(const float4* src, float4* dst, int w, int h) {
    int n = w * h;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        float4 c = src[k];
        int i = k % w, j = k / w;
        if (i >= 1 && i < w - 1 && j >= 1 && j < h - 1) {
            float l = lum(c);
            if (l > 0.0f && !(sqrtf(c.w) < 0.5f * l)) {
                float brightest = 0.0f;
                for (int dy = -1; dy <= 1; dy++)
                    for (int dx = -1; dx <= 1; dx++)
                        if (dx || dy)
                            brightest = fmaxf(brightest, lum(src[k + dy * w + dx]));
                if (l > brightest) {
                    float s = brightest / l;
                    c = make_float4(s * c.x, s * c.y, s * c.z, c.w * s * s);
                }
            }
        }
        dst[k] = c;
    }
}

// blur3x3 of the variance (denoiser.h:158-178), normalised by the weights inside the image
__global__ void k_dn_blur(const float4* L, float* bv, int w, int h) {
    int n = w * h;
    const float k3[3] = {0.25f, 0.5f, 0.25f};
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        int i = k % w, j = k / w;
        float sum = 0.0f, wt = 0.0f;
        for (int dy = -1; dy <= 1; dy++)
            for (int dx = -1; dx <= 1; dx++) {
                int x = i + dx, y = j + dy;
                if (x < 0 || x >= w || y < 0 || y >= h)
                    continue;
                float c = k3[dx + 1] * k3[dy + 1];
                sum += c * L[y * w + x].w;
                wt += c;
            }
        bv[k] = sum / wt;
    }
}

// One a-trous iteration (filter_pixel, denoiser.h:113-156) at spacing `step`.
// grid: (tiles_x * step, tiles_y * step); block (16, 16 / kRows). A thread
// filters kRows outputs, one under the other: a staged row it reads serves
// every output whose taps it holds, in each output's own order of taps. One
// output a thread was bound by shared memory (75 128-bit reads an output,
// about 62 of 100 us at 1080p); two read 45. Four read 30 but hold 94
// registers and wait more than they save (1080p frame: 805 us with one, 682
// with two, 805 with four).
constexpr int kRows = 2;
__global__ void __launch_bounds__(kTile* kTile / kRows)
    k_dn_atrous(const float4* L, const float* bv, const float4* A, const float4* N, float4* out, int w, int h, int step,
                float sigma_l, float inv_n, float inv_a) {
    __shared__ float4 sL[kSpan][kSpan];
    __shared__ float4 sA[kSpan][kSpan];
    __shared__ float4 sN[kSpan][kSpan];
    // which phase of the lattice, and which tile of that phase
    int tiles_x = (gridDim.x + step - 1) / step;  // tiles per phase column (gridDim.x = tiles_x * step)
    int phase_x = blockIdx.x / tiles_x, tile_x = blockIdx.x % tiles_x;
    int tiles_y = (gridDim.y + step - 1) / step;
    int phase_y = blockIdx.y / tiles_y, tile_y = blockIdx.y % tiles_y;
    int lx0 = tile_x * kTile - kHalo, ly0 = tile_y * kTile - kHalo;  // lattice origin of the staged span
    int tid = threadIdx.y * kTile + threadIdx.x;
    for (int e = tid; e < kSpan * kSpan; e += kTile * kTile / kRows) {
        int sx = e % kSpan, sy = e / kSpan;
        int x = phase_x + (lx0 + sx) * step, y = phase_y + (ly0 + sy) * step;
        if (x >= 0 && x < w && y >= 0 && y < h) {
            int q = y * w + x;
            sL[sy][sx] = L[q];
            sA[sy][sx] = A[q];
            sN[sy][sx] = N[q];
        } else {
            sA[sy][sx] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);  // outside the image: no tap
        }
    }
    __syncthreads();
    const int cx = threadIdx.x + kHalo, cy = threadIdx.y * kRows + kHalo;
    const int x = phase_x + (lx0 + cx) * step;
    if (x >= w || phase_x >= step || phase_y >= step)
        return;
    const float kern[5] = {1.0f / 16, 1.0f / 4, 3.0f / 8, 1.0f / 4, 1.0f / 16};
    float4 ap[kRows], np[kRows];
    float lp[kRows], inv_scale[kRows], s0[kRows], s1[kRows], s2[kRows], ws[kRows], vs[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int y = phase_y + (ly0 + cy + r) * step;
        ap[r] = sA[cy + r][cx];
        np[r] = sN[cy + r][cx];
        lp[r] = lum(sL[cy + r][cx]);
        const float scale = sigma_l * sqrtf(fmaxf(y < h ? bv[y * w + x] : 0.0f, 0.0f)) + 1e-10f;
        inv_scale[r] = 1.0f / scale;
        s0[r] = s1[r] = s2[r] = ws[r] = vs[r] = 0.0f;
    }
#pragma unroll
    for (int row = 0; row < kRows + 4; row++) {
#pragma unroll
        for (int dx = 0; dx < 5; dx++) {
            const float4 aq = sA[cy + row - 2][cx + dx - 2];
            if (aq.w < 0.0f)
                continue;
            const float4 cq = sL[cy + row - 2][cx + dx - 2], nq = sN[cy + row - 2][cx + dx - 2];
            const float lq = lum(cq);
#pragma unroll
            for (int r = 0; r < kRows; r++) {
                const int dy = row - r;  // this staged row among output r's taps
                if (dy < 0 || dy > 4)
                    continue;
                const float3 dn = f3(np[r]) - f3(nq), da = f3(ap[r]) - f3(aq);
                // which products are fused is fixed: the weights stay the same to
                // the last bit however many outputs a thread has
                const float e = fmaf(fabsf(lp[r] - lq), inv_scale[r],
                                     fmaf(dot_y(da, da), inv_a, dot_x(dn, dn) * inv_n));
                float wgt = kern[dx] * kern[dy] * __expf(-e);
                s0[r] += wgt * cq.x;
                s1[r] += wgt * cq.y;
                s2[r] += wgt * cq.z;
                ws[r] += wgt;
                vs[r] += wgt * wgt * cq.w;
            }
        }
    }
#pragma unroll
    for (int r = 0; r < kRows; r++) {
        const int y = phase_y + (ly0 + cy + r) * step;
        if (y >= h)
            continue;
        float iw = 1.0f / ws[r];
        out[y * w + x] = make_float4(s0[r] * iw, s1[r] * iw, s2[r] * iw, vs[r] * iw * iw);
    }
}

__global__ void k_dn_finish(const float4* L, const double* alb, double* out, int n) {
    const double eps = 1e-3;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        float4 c = L[k];
        out[3 * k] = double(c.x) * (alb[3 * k] + eps);
        out[3 * k + 1] = double(c.y) * (alb[3 * k + 1] + eps);
        out[3 * k + 2] = double(c.z) * (alb[3 * k + 2] + eps);
    }
}

int bad(const std::string& m) {
    set_error_message(m);
    return MYPBR_ERR_INVALID_ARGUMENT;
}

}  // namespace
}  // namespace mypbr_dev

using namespace mypbr_dev;

extern "C" void mypbr_denoise_opts_init(mypbr_denoise_opts* o) {
    if (!o)
        return;
    *o = mypbr_denoise_opts{};
    o->iterations = 5;          // denoiser.h:39-42
    o->sigma_luminance = 4;
    o->sigma_normal = 0.1;
    o->sigma_albedo = 0.1;
}

extern "C" int mypbr_gpu_denoise(const double* radiance, const double* albedo, const double* normal,
                                 const double* variance, int32_t width, int32_t height, const mypbr_denoise_opts* opts,
                                 double* out, int on_device) {
    mypbr_dev::NvtxRange range("mypbr denoise");
    if (!radiance || !albedo || !normal || !variance || !out || width < 1 || height < 1)
        return bad("mypbr_gpu_denoise: bad argument");
    mypbr_denoise_opts o;
    mypbr_denoise_opts_init(&o);
    if (opts)
        o = *opts;
    if (o.iterations < 0 || o.iterations > 16 || !(o.sigma_normal > 0) || !(o.sigma_albedo > 0))
        return bad("mypbr_gpu_denoise: iterations must be in [0, 16] and the sigmas positive");
    size_t n = size_t(width) * height;
    if (n > (size_t(1) << 30))
        return bad("mypbr_gpu_denoise: image too large");
    int dev = 0;
    MYPBR_CUDA(cudaGetDevice(&dev));
    int sms = 1;
    MYPBR_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // five planes, and with host buffers the frame in and out (Workspace keeps
    // them for the next frame: allocating and freeing them took 0.46 of a 1080p
    // frame's 1.27 ms)
    Workspace mem;
    const size_t planes = 4 * Workspace::padded<float4>(n) + Workspace::padded<float>(n);
    const size_t frame = on_device ? 0 : 4 * Workspace::padded<double>(3 * n) + Workspace::padded<double>(n);
    if (int s = mem.reserve(planes + frame); s != MYPBR_OK)
        return s;
    float4* L0 = mem.take<float4>(n);
    float4* L1 = mem.take<float4>(n);
    float4* A = mem.take<float4>(n);
    float4* N = mem.take<float4>(n);
    float* BV = mem.take<float>(n);
    const double* in[4] = {radiance, albedo, normal, variance};
    double* dst = out;
    if (!on_device) {
        size_t sizes[4] = {3 * n, 3 * n, 3 * n, n};
        for (int k = 0; k < 4; k++) {
            double* d = mem.take<double>(sizes[k]);
            if (int s = copy_to_device(d, in[k], sizes[k] * sizeof(double)); s != MYPBR_OK)
                return s;
            in[k] = d;
        }
        dst = mem.take<double>(3 * n);
    }
    int blocks = int(std::min<size_t>((n + 255) / 256, size_t(sms) * 16));
    k_dn_prepare<<<blocks, 256>>>(in[0], in[1], in[2], in[3], int(n), L0, A, N);
    k_dn_fireflies<<<blocks, 256>>>(L0, L1, width, height);
    float4* cur = L1;
    float4* nxt = L0;
    float inv_n = float(1.0 / (o.sigma_normal * o.sigma_normal)), inv_a = float(1.0 / (o.sigma_albedo * o.sigma_albedo));
    for (int it = 0; it < o.iterations; it++) {
        int step = 1 << it;
        k_dn_blur<<<blocks, 256>>>(cur, BV, width, height);
        // lattice of each phase: ceil(width / step) points wide (at most)
        int lw = (width + step - 1) / step, lh = (height + step - 1) / step;
        int tx = (lw + kTile - 1) / kTile, ty = (lh + kTile - 1) / kTile;
        dim3 grid(unsigned(tx * step), unsigned(ty * step));
        k_dn_atrous<<<grid, dim3(kTile, kTile / kRows)>>>(cur, BV, A, N, nxt, width, height, step, float(o.sigma_luminance),
                                                  inv_n, inv_a);
        std::swap(cur, nxt);
    }
    k_dn_finish<<<blocks, 256>>>(cur, in[1], dst, int(n));
    MYPBR_CUDA(cudaGetLastError());
    if (!on_device)
        return copy_to_host(out, dst, 3 * n * sizeof(double), nullptr);
    MYPBR_CUDA(cudaDeviceSynchronize());
    return MYPBR_OK;
}
