// fp32 NCHW -> int8 NHWC quantization: otter::quantize_to_int8 (Tensor/Quantize.cpp:52-58,
// Tensor/QuantizeX86.cpp:47-644) moved to the GPU, together with the layout change the reference does in
// Net::convert_layout (Tensor/Net.cpp:380-411).
//
// HBM-bound: 4 bytes read + 1 byte written per element. Each CTA moves a [64 channels x 128 pixels] tile
// of one image: reads are float4 along W (the contiguous axis of NCHW), eight of them in flight per thread, the channel/pixel
// transpose of 4x4 blocks happens in registers, 32-bit words of 4 channels go through shared memory, and writes are
// 16-byte groups of channels (the contiguous axis of NHWC). Tile coordinates are the grid's, the image of a pixel is a
// multiply-shift quotient: with 64-bit divisions a thread spent more instructions on finding its 32 elements than on them
// (17 per element; 64 channels 56x56 x256: 55.1 -> 41.6 us = 6.2 TB/s, 256 channels 28x28 x128: 31.1 -> 24.5).
#include "kernels.h"
#include "launch.cuh"

namespace ottk {

constexpr int QT_C = 64;    // channels per tile
constexpr int QT_P = 128;   // pixels per tile
constexpr int QT_THREADS = 256;
constexpr int QT_PITCH = 17;  // words per pixel row in shared memory (16 used): odd, so columns spread over banks

// pixel p of the tile lives in row (p%4)*33 + p/4: the four pixels a thread produces from one float4 land in
// four row groups, and the 32 lanes of a warp land in 32 consecutive rows of a group (no bank conflicts).
__device__ __forceinline__ int qt_row(int p) { return (p & 3) * 33 + (p >> 2); }

// A plain tensor's planes by arithmetic, a plane table's by look-up.
struct DensePlanes {
    const float* x;
    long long img_stride;
    __device__ __forceinline__ const float* plane(int c, int img, long hw) const { return x + (long long)img * img_stride + (long long)c * hw; }
};

static void advance_images(DensePlanes& g, int images) { g.x += (long long)images * g.img_stride; }
static void advance_images(PlaneGather& g, int images) {
    for (int i = 0; i < kGatherMaxBufs; ++i) g.base[i] += (long long)images * g.img_stride[i];
}

// Grid: x = pixel tile, y = channel tile, z = image (one when flat). flat: the pixel axis runs over all images (hw % 4 == 0, so a
// thread's 4 pixels never straddle two images) and no tile is wasted on the tail of an image.
template <typename Planes>
__global__ void __launch_bounds__(QT_THREADS, 4)
quantize_nchw_to_nhwc_kernel(const __grid_constant__ Planes G, int8_t* __restrict__ out, const float* __restrict__ scales, int n_scales, int c, int cpad,
                             int hw, uint32_t half, int out_stride, int flat, int vec_ok, long total_px, FastDiv div_hw) {
    __shared__ uint32_t tile[4 * 33 * QT_PITCH];
    pdl_launch_dependents();
    pdl_wait();
    const int c0 = blockIdx.y * QT_C;
    const long p0 = (long)blockIdx.x * QT_P;             // first pixel of the tile (global when flat, in-image otherwise)
    const long px_end = flat ? total_px : (long)hw;      // pixels beyond this do not exist

    // phase 1: a thread quantizes 4 consecutive pixels of 4 consecutive channels and packs, per pixel, the
    // 4 channels into one word. Lanes run along pixels (512 contiguous bytes per channel row per warp).
    constexpr int PASSES = QT_C / 32;
    const int pq = threadIdx.x & 31, cq = threadIdx.x >> 5;
    const long gp = p0 + pq * 4;
    const int img = flat ? (total_px <= 0x7FFFFFFFl ? (int)fast_div((uint32_t)gp, div_hw) : (int)(gp / hw)) : (int)blockIdx.z;
    const int p = flat ? (int)(gp - (long)img * hw) : (int)gp;
    const bool vec = vec_ok && gp + 3 < px_end;
    float4 v[PASSES][4];
#pragma unroll
    for (int pass = 0; pass < PASSES; ++pass)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int cg = c0 + (cq + 8 * pass) * 4 + i;
            v[pass][i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (cg < c) {
                const float* row = G.plane(cg, img, hw) + p;
                if (vec) {
                    v[pass][i] = __ldg(reinterpret_cast<const float4*>(row));
                } else {
                    if (gp < px_end) v[pass][i].x = __ldg(row);
                    if (gp + 1 < px_end) v[pass][i].y = __ldg(row + 1);
                    if (gp + 2 < px_end) v[pass][i].z = __ldg(row + 2);
                    if (gp + 3 < px_end) v[pass][i].w = __ldg(row + 3);
                }
            }
        }
#pragma unroll
    for (int pass = 0; pass < PASSES; ++pass) {
        const int cword = cq + 8 * pass;
        if (c0 + cword * 4 >= cpad) break;  // narrow tensors: nothing of these channels is ever stored
        uint32_t cw[4];  // channel i: its 4 pixels packed
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int cg = c0 + cword * 4 + i;
            const float sc = n_scales == 1 ? __ldg(scales) : (cg < c ? __ldg(scales + cg) : 0.f);
            cw[i] = quantize4_pack(v[pass][i].x, v[pass][i].y, v[pass][i].z, v[pass][i].w, sc, half);
        }
        uint32_t pw[4];  // pixel j: its 4 channels packed
        transpose4x4(cw[0], cw[1], cw[2], cw[3], pw);
#pragma unroll
        for (int j = 0; j < 4; ++j) tile[(j * 33 + pq) * QT_PITCH + cword] = pw[j];
    }
    __syncthreads();
    // phase 2: 16-byte channel groups; consecutive threads -> consecutive groups of one pixel
    int8_t* dst = out + ((flat ? 0l : (long)blockIdx.z * hw) + p0) * out_stride + c0;
#pragma unroll
    for (int i = threadIdx.x; i < QT_P * (QT_C / 16); i += QT_THREADS) {
        const int pl = i >> 2, g = i & 3;
        if (p0 + pl < px_end && c0 + g * 16 < cpad) {
            const uint32_t* r = tile + qt_row(pl) * QT_PITCH + g * 4;
            *reinterpret_cast<uint4*>(dst + (long)pl * out_stride + g * 16) = make_uint4(r[0], r[1], r[2], r[3]);
        }
    }
}

template <typename Planes>
static cudaError_t launch_quantize(cudaStream_t stream, const Planes& src, int8_t* out, int out_stride, const float* scales_dev, int n_scales, int vec_ok,
                                   int n, int c, int cpad, int hw, int rounding) {
    const int flat = hw % 4 == 0 ? 1 : 0;
    const long total_px = (long)n * hw, span = flat ? total_px : hw;
    for (int img0 = 0; img0 < (flat ? 1 : n); img0 += 65535) {  // (the grid's third dimension ends at 65535)
        Planes part = src;
        if (img0 > 0) advance_images(part, img0);
        const dim3 grid((unsigned)((span + QT_P - 1) / QT_P), (unsigned)((cpad + QT_C - 1) / QT_C), (unsigned)(flat ? 1 : (n - img0 < 65535 ? n - img0 : 65535)));
        const cudaError_t e = launch_overlapped(quantize_nchw_to_nhwc_kernel<Planes>, grid, dim3(QT_THREADS), 0, stream, part, out + (long)img0 * hw * out_stride,
                                                scales_dev, n_scales, c, cpad, hw, half_bits(rounding), out_stride, flat, vec_ok, total_px,
                                                make_fast_div((uint32_t)hw));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void gather_identity(PlaneGather* g, const float* x, int c, int c_total, long hw) {
    g->base[0] = x;
    g->img_stride[0] = (long long)c_total * hw;
    for (int i = 0; i < c && i < kGatherMaxChannels; ++i) g->ref[i] = (uint32_t)i;
}

cudaError_t launch_quantize_nchw_to_nhwc(cudaStream_t stream, const PlaneGather& src, int8_t* out, const float* scales_dev,
                                         int n_scales, int n, int c, int h, int w, int rounding) {
    const int hw = h * w, cpad = nhwc_channels(c);
    if (n == 0 || hw == 0) return cudaSuccess;
    if (c > kGatherMaxChannels) return cudaErrorInvalidValue;
    bool aligned = hw % 4 == 0;  // four pixels of a plane are one 16-byte load
    for (int i = 0, last = -1; i < c && aligned; ++i) {
        const int b = (int)(src.ref[i] >> 24);
        if (b != last) aligned = (reinterpret_cast<uintptr_t>(src.base[b]) & 15) == 0 && src.img_stride[b] % 4 == 0;
        last = b;
    }
    return launch_quantize(stream, src, out, cpad, scales_dev, n_scales, aligned ? 1 : 0, n, c, cpad, hw, rounding);
}

// a plain tensor of any channel count
cudaError_t launch_quantize_dense(cudaStream_t stream, const float* x, int c_total, int8_t* out, const float* scales_dev, int n_scales,
                                  int n, int c, int h, int w, int rounding) {
    const int hw = h * w, cpad = nhwc_channels(c);
    if (n == 0 || hw == 0) return cudaSuccess;
    return launch_quantize(stream, DensePlanes{x, (long long)c_total * hw}, out, cpad, scales_dev, n_scales,
                           hw % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? 1 : 0, n, c, cpad, hw, rounding);
}

// dst[img][c][p] = plane(c, img)[p]
__global__ void gather_planes_kernel(const __grid_constant__ PlaneGather G, float* __restrict__ dst, int c, long hw, long total4, int vec) {
    pdl_launch_dependents();
    pdl_wait();
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += (long)gridDim.x * blockDim.x) {
        const long per = vec ? hw / 4 : hw;
        const long p = i % per;
        const long r = i / per;
        const int ch = (int)(r % c);
        const int img = (int)(r / c);
        const float* src = G.plane(ch, img, hw);
        if (vec) reinterpret_cast<float4*>(dst)[i] = __ldg(reinterpret_cast<const float4*>(src) + p);
        else dst[i] = __ldg(src + p);
    }
}

// dst[img][c][p] = A.plane(c, img)[p] + B.plane(c, img)[p]: the reference's ShortCut (Tensor/ShortCutLayer.cpp) reading both
// operands where their planes lie. Block = one plane (or a slice of one), so the table look-up is per block, not per element.
__global__ void add_planes_kernel(const __grid_constant__ PlaneGather A, const __grid_constant__ PlaneGather B, float* __restrict__ dst, int c,
                                  long hw, int slices, int vec) {
    pdl_launch_dependents();
    pdl_wait();
    const long plane = blockIdx.x / slices;
    const int slice = (int)(blockIdx.x % slices);
    const int ch = (int)(plane % c);
    const int img = (int)(plane / c);
    const float* a = A.plane(ch, img, hw);
    const float* b = B.plane(ch, img, hw);
    float* o = dst + plane * hw;
    const long per = vec ? hw / 4 : hw;
    const long lo = per * slice / slices, hi = per * (slice + 1) / slices;
    if (vec) {
        for (long i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            const float4 u = __ldg(reinterpret_cast<const float4*>(a) + i), v = __ldg(reinterpret_cast<const float4*>(b) + i);
            reinterpret_cast<float4*>(o)[i] = make_float4(__fadd_rn(u.x, v.x), __fadd_rn(u.y, v.y), __fadd_rn(u.z, v.z), __fadd_rn(u.w, v.w));
        }
    } else {
        for (long i = lo + threadIdx.x; i < hi; i += blockDim.x) o[i] = __fadd_rn(__ldg(a + i), __ldg(b + i));
    }
}

cudaError_t launch_add_planes(cudaStream_t stream, const PlaneGather& a, const PlaneGather& b, float* dst, int n, int c, long hw) {
    if (n == 0 || c == 0 || hw == 0) return cudaSuccess;
    if (c > kGatherMaxChannels) return cudaErrorInvalidValue;
    const int vec = hw % 4 == 0 ? 1 : 0;
    const long per = vec ? hw / 4 : hw;
    const int threads = per >= 256 ? 256 : (per >= 128 ? 128 : 64);
    int slices = (int)((per + 4L * threads - 1) / (4L * threads));  // about four elements (vectors) per thread
    if (slices < 1) slices = 1;
    const long blocks = (long)n * c * slices;
    if (blocks > 0x7fffffffL) return cudaErrorInvalidValue;
    return launch_overlapped(add_planes_kernel, dim3((unsigned)blocks), dim3(threads), 0, stream, a, b, dst, c, hw, slices, vec);
}

cudaError_t launch_gather_planes(cudaStream_t stream, const PlaneGather& src, float* dst, int n, int c, long hw) {
    if (n == 0 || c == 0 || hw == 0) return cudaSuccess;
    if (c > kGatherMaxChannels) return cudaErrorInvalidValue;
    const int vec = hw % 4 == 0 ? 1 : 0;
    const long total = (long)n * c * (vec ? hw / 4 : hw);
    long grid = (total + 255) / 256;
    if (grid > 148 * 16) grid = 148 * 16;
    return launch_overlapped(gather_planes_kernel, dim3((unsigned)grid), dim3(256), 0, stream, src, dst, c, hw, total, vec);
}

}  // namespace ottk
