// First-layer ("stem") int8 convolution: 3 input channels, 3x3, stride 1 or 2, fp32 NCHW image in, with the
// quantize prologue (Tensor/QuantizeX86.cpp:47-644) and the dequantize/requantize epilogue fused.
// Reference kernels: conv2d_3x3s2_int8_pack1to4 (Tensor/ConvolutionMM2DInt8X86Pack.cpp:2569-2651) and the generic
// pack1to4 im2col path (:2225-2261).
//
// HBM-bound (12 B of image per input pixel in, Cout*4 or Cout bytes per output pixel out). One CTA computes a
// 32x8 tile of output pixels for all output channels:
//  1. the fp32 input halo tile is quantized once into shared memory as int8 channel planes;
//  2. each thread gathers the 27 taps of its output pixel into 7 registers (4 taps per register, K order
//     channel-row-column) with funnel shifts and byte permutes;
//  3. 7 dp4a per output channel against the packed filter, which lives in the kernel parameter bank so every
//     multiply reads its weights as an immediate constant operand (warp-uniform, no loads);
//  4. epilogue per channel; fp32 NCHW stores are coalesced along the tile row, int8 NHWC stores are 16-byte vectors.
#include "launch.cuh"
#include "store.cuh"
#include "umma_primitives.cuh"

namespace ottk {

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
    static const EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(p);
        return nullptr;
    }();
    return fn;
}

constexpr int ST_TX = 32, ST_TY = 8;  // output tile
constexpr int ST_COUT_MAX = 32;

struct StemParams {
    uint32_t w[ST_COUT_MAX][7];  // packed filters: byte k of the 28 = tap (c, ky, kx) with k = c*9 + ky*3 + kx
    float scale_in[ST_COUT_MAX], bias[ST_COUT_MAX], scale_out[ST_COUT_MAX];
};

template <int S, int OUT, int ACT>
__global__ void __launch_bounds__(ST_TX * ST_TY)
dense_stem_kernel(const float* __restrict__ x, const __grid_constant__ StemParams P, float in_scale, int has_bias, float act_p0,
                  uint32_t half, void* __restrict__ out, ConvShape s, int tiles_x, int tiles_y) {
    constexpr int IW = (ST_TX - 1) * S + 3, IH = (ST_TY - 1) * S + 3;  // input halo tile
    constexpr int RP = (IW + 3 + 3) / 4 + 1;                            // words per row (tile origin rounded down to 4)
    __shared__ uint32_t tin[3][IH][RP];

    int b = blockIdx.x;
    const int tx = b % tiles_x; b /= tiles_x;
    const int ty = b % tiles_y;
    const int img = b / tiles_y;
    const int ox0 = tx * ST_TX, oy0 = ty * ST_TY;
    const int iy0 = oy0 * S - s.ph, ix_first = ox0 * S - s.pw;
    const int ix_al = (ix_first >= 0 ? ix_first : ix_first - 3) / 4 * 4;
    const int sh = ix_first - ix_al;  // 0..3

    // ---- 1. quantize the halo tile ----
    const float* ximg = x + (long)img * 3 * s.h * s.w;
    const bool vec_ok = s.w % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;  // four pixels are one 16-byte load
    for (int i = threadIdx.x; i < 3 * IH * RP; i += ST_TX * ST_TY) {
        const int xw = i % RP, r = (i / RP) % IH, c = i / (RP * IH);
        const int iy = iy0 + r, ix = ix_al + xw * 4;
        uint32_t word = 0;
        if (iy >= 0 && iy < s.h && ix + 3 >= 0 && ix < s.w) {
            const float* row = ximg + ((long)c * s.h + iy) * s.w;
            if (vec_ok && ix >= 0 && ix + 3 < s.w) {
                const float4 v = __ldg(reinterpret_cast<const float4*>(row + ix));
                word = quantize4_pack(v.x, v.y, v.z, v.w, in_scale, half);
            } else {
                int q[4] = {0, 0, 0, 0};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (ix + j >= 0 && ix + j < s.w) q[j] = quantize1(__ldg(row + ix + j), in_scale, half);
                word = pack4(q[0], q[1], q[2], q[3]);
            }
        }
        tin[c][r][xw] = word;
    }
    __syncthreads();

    // ---- 2. gather the 27 taps of this thread's pixel ----
    const int lx = threadIdx.x % ST_TX, ly = threadIdx.x / ST_TX;
    const int ox = ox0 + lx, oy = oy0 + ly;
    const int boff = sh + lx * S;  // byte offset of the pixel's first tap column in a tile row
    const int wi = boff >> 2, bs = (boff & 3) * 8;
    uint32_t win[9];  // (c, ky): bytes 0..2 = taps kx 0..2
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
            const uint32_t* p = &tin[c][ly * S + ky][wi];
            win[c * 3 + ky] = __funnelshift_r(p[0], p[1], bs);
        }
    // K words: byte k = win[k / 3] byte (k % 3)
    uint32_t kw[7];
    kw[0] = __byte_perm(win[0], win[1], 0x4210);  // k0..3  = w0.b0 w0.b1 w0.b2 w1.b0
    kw[1] = __byte_perm(win[1], win[2], 0x5421);  // k4..7  = w1.b1 w1.b2 w2.b0 w2.b1
    kw[2] = __byte_perm(win[2], win[3], 0x6542);  // k8..11 = w2.b2 w3.b0 w3.b1 w3.b2
    kw[3] = __byte_perm(win[4], win[5], 0x4210);
    kw[4] = __byte_perm(win[5], win[6], 0x5421);
    kw[5] = __byte_perm(win[6], win[7], 0x6542);
    kw[6] = __byte_perm(win[8], 0u, 0x4210);      // k24..26, byte 3 = 0

    // ---- 3. multiply + 4. epilogue ----
    const bool valid = ox < s.ow && oy < s.oh;
    const long oplane = (long)s.oh * s.ow;
    float* of32 = reinterpret_cast<float*>(out) + (long)img * s.cout * oplane + (long)oy * s.ow + ox;
    int8_t* os8 = reinterpret_cast<int8_t*>(out) + (((long)img * s.oh + oy) * s.ow + ox) * s.cout_pad;
#pragma unroll
    for (int g = 0; g < ST_COUT_MAX / 4; ++g) {
        if (g * 4 >= s.cout_pad) break;
        int qv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int co = g * 4 + j;
            int acc = 0;
#pragma unroll
            for (int k = 0; k < 7; ++k) acc = __dp4a((int)kw[k], (int)P.w[co][k], acc);
            const float a = __int2float_rn(acc);
            float v = has_bias ? __fmaf_rn(a, P.scale_in[co], P.bias[co]) : __fmul_rn(a, P.scale_in[co]);
            v = activate_t<ACT>(v, act_p0);
            if (OUT == DT_F32_NCHW) {
                if (valid && co < s.cout) of32[(long)co * oplane] = v;
            } else {
                qv[j] = float2int8(__fmul_rn(v, P.scale_out[co]), half);
            }
        }
        if (OUT == DT_S8_NHWC && valid) *reinterpret_cast<uint32_t*>(os8 + g * 4) = pack4(qv[0], qv[1], qv[2], qv[3]);
    }
}

// ---- stem convolution followed by a 3x3 stride-2 pad-1 max-pool, in one kernel ----
// The pool is the only consumer of the first layer's output in the benchmark graphs (conv1 -> pool1), and that output is
// the largest tensor of the whole network; here it never leaves the SM. One CTA produces a tile of 16 x 6 POOLED pixels for all
// channels, as eight patches of 4 x 3: warp w has patch (w % 4, w / 4), i.e. the 9 x 7 convolution outputs under it.
// pad_zero selects the reference's packed max-pool rule (padding counts as 0, Tensor/Pool.cpp:972-975) or its plain
// rule (padding never wins).
constexpr int SP_PX = 16, SP_PY = 6;                         // pooled tile
constexpr int SP_CX = 2 * SP_PX + 1, SP_CY = 2 * SP_PY + 1;  // convolution outputs under it
constexpr int SP_PW = 9, SP_PH = 7, SP_ROWS = 64;            // convolution outputs of a patch, 63 and a row nobody reads

// The multiply-adds run on the tensor cores with channels as accumulator rows. A convolution pixel's 27 taps, gathered into 7 registers
// with funnel shifts and byte permutes exactly as in the kernel above, are 32 bytes of a shared-memory row; a row has those of the same
// pixel of four patches side by side (K = 128), and the filters stand four times on the diagonal of a 128 x 128 matrix, so that
// D[32 g + channel, pixel] = filter(channel) * taps(patch g, pixel): three quarters of the products are with zeros, which the tensor pipe has
// to spare (four MMAs, 256 cycles per CTA). Warp g of a lane quarter then holds one channel per lane and the pixels of ONE patch as
// columns: the pool is 40 three-way maxima of its own registers, the epilogue's parameters are three registers, and nothing of the 495
// accumulators goes through shared memory (which it did, 16 bytes at a time, at two thirds of what that pipe delivers). The fp32 halo
// tile comes as one TMA box, zeros outside the image included, and is quantized word by word in the order it lies. The CTAs stay (four per
// SM) and set the filter matrix and tensor memory up once; the next tile's box comes while this one is pooled. 24 channels, 320x320 x256, int8
// out: 212 us with pixels as rows, an index calculation per loaded word and a CTA per tile; 174 with channels as rows and boxes, 151 with CTAs
// that stay (48 at the copy rate). What is left is issue slots (half of them), spread over the phases.
//
// OUT8: the pooled values leave quantized, float2int8(v * scale_out[channel]), as an int8 NHWC tensor (what the quantize pass of
// the layers reading the pooled blob would compute from the fp32 values) instead of fp32 NCHW planes. A warp's four neighbouring
// pooled pixels of 32 channels leave as 128 consecutive bytes.
template <int S>
struct StemTile {
    static constexpr int IH = (SP_CY - 1) * S + 3;                  // input rows
    static constexpr int RP = ((SP_CX - 1) * S + 3 + 3) / 4 + 1;    // words of four pixels in a row (tile origin rounded down to 4)
    static constexpr int WORDS = 3 * IH * RP;
    // filter matrix, then the fp32 words and later, over them, the rows of taps, then the quantized words
    static constexpr int TAPS = 16384, REGION = TAPS + (WORDS * 16 > 16384 ? (WORDS * 16 + 1023) / 1024 * 1024 : 16384), BYTES = REGION + WORDS * 4;
};

template <int S, int ACT, bool OUT8>
__global__ void __launch_bounds__(256, 4)
dense_stem_pool_mma_kernel(const __grid_constant__ CUtensorMap image, const float* __restrict__ x, const __grid_constant__ StemParams P, float in_scale, float act_p0,
                           uint32_t half, void* __restrict__ out_any, ConvShape s, int ph_out, int pw_out, int tiles_x, int tiles_y, int tiles, FastDiv div_x, FastDiv div_y,
                           int by_box, int pad_zero, uint32_t* __restrict__ status, unsigned long long wait_ns) {
    using namespace umma;
    using Tile = StemTile<S>;
    constexpr int IH = Tile::IH, RP = Tile::RP, WORDS = Tile::WORDS;
    extern __shared__ uint8_t smem_spm[];
    const uint32_t base = (smem_u32(smem_spm) + 1023u) & ~1023u;
    uint8_t* bp = smem_spm + (base - smem_u32(smem_spm));
    uint8_t* sW = bp;               // [128][128 B]: the filters on the diagonal, 128-byte swizzle
    uint8_t* sT = bp + Tile::TAPS;  // [128][128 B]: pixel 64 (patch / 4) + i of patches 0..3 or 4..7, 128-byte swizzle
    uint32_t* tin = reinterpret_cast<uint32_t*>(bp + Tile::REGION);  // [3][IH][RP] int8 channel planes
    __shared__ __align__(16) float sprm[3][ST_COUT_MAX];  // scale_in, bias, scale_out
    __shared__ __align__(8) unsigned long long bar_storage[2];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_flag;
    const uint32_t bar_x = smem_u32(&bar_storage[0]), bar_d = smem_u32(&bar_storage[1]);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // where a tile lies: its image, first pooled pixel, and the word its first input column lies in
    struct Place {
        int img, px0, py0, ix_al;
    };
    const auto locate = [&](int t) {
        const int row = (int)fast_div((uint32_t)t, div_x), img = (int)fast_div((uint32_t)row, div_y), px0 = (t - row * tiles_x) * SP_PX;
        const int ix = (2 * px0 - 1) * S - s.pw;  // (pool pad 1)
        return Place{img, px0, (row - img * tiles_y) * SP_PY, (ix >= 0 ? ix : ix - 3) / 4 * 4};
    };
    const auto fetch = [&](int t) {
        const Place a = locate(t);
        mbar_expect_tx(bar_x, (uint32_t)WORDS * 16u);
        tma_load_4d(&image, bar_x, base + Tile::TAPS, a.ix_al, (2 * a.py0 - 1) * S - s.ph, 0, a.img);
    };

    if (warp == 7) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(128u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        pdl_launch_dependents();  // not before this CTA has its tensor memory: see dense_umma.cu
    }
    if (threadIdx.x == 0) {
        mbar_init(bar_x, 1);
        mbar_init(bar_d, 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (by_box) {
            pdl_wait();
            fetch((int)blockIdx.x);
        }
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + ST_COUT_MAX) {
        const int o = threadIdx.x - 64;
        sprm[0][o] = P.scale_in[o];
        sprm[1][o] = P.bias[o];
        sprm[2][o] = P.scale_out[o];
    }
    // filter matrix: row 32 g + channel, 28 bytes of taps and 4 of zeros at byte 32 g
    {
        const int row = threadIdx.x >> 1, j = threadIdx.x & 1;
#pragma unroll
        for (int d = 1; d < 4; ++d) {
            const int chunk = 2 * (((row >> 5) + d) & 3) + j;
            *reinterpret_cast<uint4*>(sW + row * 128 + ((chunk ^ (row & 7)) << 4)) = make_uint4(0, 0, 0, 0);
        }
        if (threadIdx.x < 64) {
            const uint4 w4 = j == 0 ? make_uint4(P.w[row][0], P.w[row][1], P.w[row][2], P.w[row][3]) : make_uint4(P.w[row][4], P.w[row][5], P.w[row][6], 0u);
#pragma unroll
            for (int g = 0; g < 4; ++g) *reinterpret_cast<uint4*>(sW + (32 * g + row) * 128 + (((2 * g + j) ^ (row & 7)) << 4)) = w4;
        }
    }
    __syncthreads();
    pdl_wait();  // set-up above overlaps the previous kernel; the image is read and the output written after it
    const uint32_t tmem_base = tmem_slot;
    const int c = lane, g = warp & 3, row3 = 3 * (warp >> 2);  // this thread's channel, its warp's patch: pooled columns 4 g .. 4 g + 3, rows row3 .. row3 + 2
    const float p_si = sprm[0][c], p_bi = sprm[1][c], p_so = sprm[2][c];
    bool ok = true;
    uint32_t phase = 0;
    for (int t = (int)blockIdx.x; t < tiles; t += (int)gridDim.x, phase ^= 1u) {
    if (by_box) {
        if (!mbar_wait_warp(bar_x, phase, &abort_flag, status, 32u, wait_ns)) {
            ok = false;
            const unsigned long long t0 = globaltimer_ns();
            while (globaltimer_ns() - t0 < 1000000ull) {}  // let the copy in flight land before its place is written
        }
#pragma unroll 2
        for (int i = threadIdx.x; i < WORDS; i += 256) {
            const float4 v = reinterpret_cast<const float4*>(sT)[i];
            tin[i] = quantize4_pack(v.x, v.y, v.z, v.w, in_scale, half);
        }
    } else {
        const Place a = locate(t);
        const float* ximg = x + (long)a.img * 3 * s.h * s.w;
        const int iy0 = (2 * a.py0 - 1) * S - s.ph, ix_al = a.ix_al;
        for (int i = threadIdx.x; i < WORDS; i += 256) {
            const int xw = i % RP, r = (i / RP) % IH, c = i / (RP * IH);
            const int iy = iy0 + r, ix = ix_al + xw * 4;
            uint32_t word = 0;
            if (iy >= 0 && iy < s.h && ix + 3 >= 0 && ix < s.w) {
                const float* row = ximg + ((long)c * s.h + iy) * s.w;
                int q[4] = {0, 0, 0, 0};
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (ix + j >= 0 && ix + j < s.w) q[j] = quantize1(__ldg(row + ix + j), in_scale, half);
                word = pack4(q[0], q[1], q[2], q[3]);
            }
            tin[i] = word;
        }
    }
    __syncthreads();

    const Place at = locate(t);
    // rows of taps (byte k = tap (c, ky, kx), k = c*9 + ky*3 + kx)
#pragma unroll
    for (int rep = 0; rep < 2; ++rep) {
        const int p = threadIdx.x + 256 * rep, patch = p / SP_ROWS, i = p % SP_ROWS, g = patch & 3, n = (patch >> 2) * SP_ROWS + i;
        if (i < SP_PW * SP_PH) {
            const int lx = 8 * g + i % SP_PW, ly = 6 * (patch >> 2) + i / SP_PW;
            const int boff = (2 * at.px0 - 1 + lx) * S - s.pw - at.ix_al;
            const int wi = boff >> 2, bs = (boff & 3) * 8;
            const uint32_t* t0 = tin + ly * S * RP + wi;
            uint32_t win[9];
#pragma unroll
            for (int c = 0; c < 3; ++c)
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) {
                    const uint32_t* q = t0 + (c * IH + ky) * RP;
                    win[c * 3 + ky] = __funnelshift_r(q[0], q[1], bs);
                }
            uint4 c0, c1;
            c0.x = __byte_perm(win[0], win[1], 0x4210);
            c0.y = __byte_perm(win[1], win[2], 0x5421);
            c0.z = __byte_perm(win[2], win[3], 0x6542);
            c0.w = __byte_perm(win[4], win[5], 0x4210);
            c1.x = __byte_perm(win[5], win[6], 0x5421);
            c1.y = __byte_perm(win[6], win[7], 0x6542);
            c1.z = __byte_perm(win[8], 0u, 0x4210);
            c1.w = 0u;
            *reinterpret_cast<uint4*>(sT + n * 128 + (((2 * g) ^ (n & 7)) << 4)) = c0;
            *reinterpret_cast<uint4*>(sT + n * 128 + (((2 * g + 1) ^ (n & 7)) << 4)) = c1;
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // generic-proxy writes -> visible to the MMA's reads
    tc_fence_before();
    __syncthreads();
    tc_fence_after();

    if (warp == 1) {
        if (elect_one()) {
            // D = s32, A = B = signed int8, both K-major, N = 128, M = 128
            const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
            const uint64_t wdesc = make_smem_desc(smem_u32(sW), 128), tdesc = make_smem_desc(smem_u32(sT), 128);
#pragma unroll
            for (int k = 0; k < 4; ++k) umma_i8(tmem_base, wdesc + 2u * k, tdesc + 2u * k, idesc, k != 0 ? 1u : 0u);
            umma_commit(bar_d);
        }
        __syncwarp();
    }
    if (!mbar_wait_warp(bar_d, phase, &abort_flag, status, 32u, wait_ns)) ok = false;
    tc_fence_after();
    // the next tile's box takes the place of the taps, which the MMAs have read, while this tile is pooled
    if (by_box && threadIdx.x == 0 && ok && t + (int)gridDim.x < tiles) fetch(t + (int)gridDim.x);
    __syncwarp();

    if (ok) {
        // Max-pooling happens on the exact s32 sums: dequantize + activation is non-decreasing in the sum for the non-negative scales the
        // layer is prepared with, so the maximum of the window's outputs is the output of the window's maximum, bit for bit, and the
        // float epilogue runs once per pooled value instead of once per convolution output. Pixels outside the image never win.
        const int ox0 = 2 * at.px0 - 1 + 8 * g, oy0 = 2 * at.py0 - 1 + 2 * row3;  // the patch's first convolution output
        const bool edge = ox0 < 0 || oy0 < 0 || ox0 + SP_PW > s.ow || oy0 + SP_PH > s.oh;  // (uniform)
        const uint32_t taddr = tmem_base + ((uint32_t)(g * 32) << 16) + (uint32_t)((warp >> 2) * SP_ROWS);
        int h[SP_PH][4], rest[5];  // maxima of three neighbours in a row; the start of a row that the first 32 columns cut
        auto inside = [&](int i) { return (unsigned)(ox0 + i % SP_PW) < (unsigned)s.ow && (unsigned)(oy0 + i / SP_PW) < (unsigned)s.oh; };
        {
            int v[32];
            tmem_ld16(taddr, *reinterpret_cast<int(*)[16]>(&v[0]));
            tmem_ld16(taddr + 16u, *reinterpret_cast<int(*)[16]>(&v[16]));
            tmem_wait_ld16(*reinterpret_cast<int(*)[16]>(&v[0]));
            tmem_wait_ld16(*reinterpret_cast<int(*)[16]>(&v[16]));
            if (edge)
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (!inside(i)) v[i] = INT_MIN;
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k) h[r][k] = __vimax3_s32(v[r * 9 + 2 * k], v[r * 9 + 2 * k + 1], v[r * 9 + 2 * k + 2]);
#pragma unroll
            for (int j = 0; j < 5; ++j) rest[j] = v[27 + j];
        }
        {
            int v[32];
            tmem_ld16(taddr + 32u, *reinterpret_cast<int(*)[16]>(&v[0]));
            tmem_ld16(taddr + 48u, *reinterpret_cast<int(*)[16]>(&v[16]));
            tmem_wait_ld16(*reinterpret_cast<int(*)[16]>(&v[0]));
            tmem_wait_ld16(*reinterpret_cast<int(*)[16]>(&v[16]));
            if (edge)
#pragma unroll
                for (int i = 0; i < 31; ++i)
                    if (!inside(32 + i)) v[i] = INT_MIN;
            h[3][0] = __vimax3_s32(rest[0], rest[1], rest[2]);
            h[3][1] = __vimax3_s32(rest[2], rest[3], rest[4]);
            h[3][2] = __vimax3_s32(rest[4], v[0], v[1]);
            h[3][3] = __vimax3_s32(v[1], v[2], v[3]);
#pragma unroll
            for (int r = 4; r < SP_PH; ++r)
#pragma unroll
                for (int k = 0; k < 4; ++k) h[r][k] = __vimax3_s32(v[r * 9 - 32 + 2 * k], v[r * 9 - 31 + 2 * k], v[r * 9 - 30 + 2 * k]);
        }
        const int px = at.px0 + 4 * g;
        const long pplane = (long)ph_out * pw_out;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int py = at.py0 + row3 + r;
            float y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int m = __vimax3_s32(h[2 * r][k], h[2 * r + 1][k], h[2 * r + 2][k]);
                y[k] = activate_t<ACT>(__fmaf_rn(__int2float_rn(m), p_si, p_bi), act_p0);
                if (ACT != ACT_RELU && ACT != ACT_RELU6) {  // (after a ReLU nothing is below the padding's 0)
                    // the reference's packed max-pool lets the padding take part as 0 (Tensor/Pool.cpp:972-975); its plain one never lets it win
                    const int cx = 2 * (px + k) - 1, cy = 2 * py - 1;
                    if (pad_zero && (cx < 0 || cx + 2 >= s.ow || cy < 0 || cy + 2 >= s.oh)) y[k] = fmaxf(y[k], 0.f);
                }
            }
            if (OUT8) {
                const int2 a = round2(__fmul2_rn(make_float2(y[0], y[1]), make_float2(p_so, p_so)), half);
                const int2 e = round2(__fmul2_rn(make_float2(y[2], y[3]), make_float2(p_so, p_so)), half);
                uint32_t w = c < s.cout ? pack_sat_s8x4(a.x, a.y, e.x, e.y) : 0u;
                // 4x4 byte transpose across four lanes: lane 4 k + p then holds pixel p's channels 4 k .. 4 k + 3
                const int p = lane & 3;
                w = __byte_perm(w, __shfl_xor_sync(0xFFFFFFFFu, w, 2), p < 2 ? 0x5410u : 0x3276u);
                w = __byte_perm(w, __shfl_xor_sync(0xFFFFFFFFu, w, 1), (p & 1) == 0 ? 0x6240u : 0x3715u);
                const int cq = lane & ~3;
                if (py < ph_out && px + p < pw_out && cq < s.cout_pad)
                    *reinterpret_cast<uint32_t*>(static_cast<int8_t*>(out_any) + (((long)at.img * ph_out + py) * pw_out + px + p) * s.cout_pad + cq) = w;
            } else if (py < ph_out && c < s.cout) {
                float* o = static_cast<float*>(out_any) + ((long)at.img * s.cout + c) * pplane + (long)py * pw_out + px;
                if (px + 3 < pw_out && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
                    *reinterpret_cast<float4*>(o) = make_float4(y[0], y[1], y[2], y[3]);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (px + k < pw_out) o[k] = y[k];
                }
            }
        }
    }
    tc_fence_before();  // (the next tile's MMAs come after the barriers below its loads)
    }
    __syncthreads();
    if (warp == 7) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(128u) : "memory");
    }
}

template <int S, int OUT>
cudaError_t launch_act(cudaStream_t stream, const float* x, const StemParams& P, float in_scale, const EpilogueParams& ep, void* out,
                       const ConvShape& s) {
    const int tiles_x = (s.ow + ST_TX - 1) / ST_TX, tiles_y = (s.oh + ST_TY - 1) / ST_TY;
    const long blocks = (long)s.n * tiles_x * tiles_y;
    if (blocks == 0) return cudaSuccess;
    const dim3 grid((unsigned)blocks), block(ST_TX * ST_TY);
#define OTT_STEM_LAUNCH(ACT) \
    dense_stem_kernel<S, OUT, ACT><<<grid, block, 0, stream>>>(x, P, in_scale, ep.has_bias, ep.act_param0, half_bits(ep.rounding), out, s, tiles_x, tiles_y)
    switch (ep.act_type) {
        case ACT_RELU: OTT_STEM_LAUNCH(ACT_RELU); break;
        case ACT_LRELU: OTT_STEM_LAUNCH(ACT_LRELU); break;
        case ACT_RELU6: OTT_STEM_LAUNCH(ACT_RELU6); break;
        default: OTT_STEM_LAUNCH(ACT_NONE); break;
    }
#undef OTT_STEM_LAUNCH
    return cudaGetLastError();
}

}  // namespace

bool dense_stem_supports(const ConvShape& s, int in_dtype, int out_dtype) {
    return in_dtype == DT_F32_NCHW && (out_dtype == DT_F32_NCHW || out_dtype == DT_S8_NHWC) && s.cin == 3 && s.kh == 3 && s.kw == 3 &&
           s.dh == 1 && s.dw == 1 && s.sh == s.sw && (s.sh == 1 || s.sh == 2) && s.cout_pad <= ST_COUT_MAX;
}

static void fill_stem_params(StemParams& P, const ConvShape& s, const int8_t* w, const float* scale_in, const float* bias, const float* scale_out) {
    for (int o = 0; o < s.cout; ++o) {
        // The kernels assume scale_in >= 0 (it is 1 / (positive scales)). Should one ever be negative, the channel's filter and
        // scale are negated together: (-acc) * (-scale) is the same product, exactly.
        const int sign = scale_in[o] < 0.f ? -1 : 1;
        for (int k = 0; k < 27; ++k) P.w[o][k / 4] |= (uint32_t)(uint8_t)(int8_t)(sign * w[o * 27 + k]) << (8 * (k % 4));
        P.scale_in[o] = sign * scale_in[o];
        P.bias[o] = bias ? bias[o] : 0.f;
        P.scale_out[o] = scale_out ? scale_out[o] : 0.f;
    }
}

template <int S, bool OUT8>
static cudaError_t launch_pool_s(cudaStream_t stream, const float* x, const StemParams& P, float in_scale, const EpilogueParams& ep, void* out,
                                 const ConvShape& s, int pad_zero, uint32_t* status, int sm_count, unsigned long long wait_ns) {
    using Tile = StemTile<S>;
    const int ph_out = (s.oh + 2 - 3) / 2 + 1, pw_out = (s.ow + 2 - 3) / 2 + 1;
    const int tiles_x = (pw_out + SP_PX - 1) / SP_PX, tiles_y = (ph_out + SP_PY - 1) / SP_PY;
    const long blocks = (long)s.n * tiles_x * tiles_y;
    if (blocks <= 0) return cudaSuccess;
    if (blocks > 0x7FFFFFFFl) return cudaErrorInvalidValue;
    const long resident = 4l * sm_count;  // CTAs of the whole GPU at once; each walks over its tiles
    // the halo tile as one box: rows of whole 16-byte words from a 16-byte boundary; any other image pixel by pixel
    CUtensorMap image{};
    const int by_box = s.w % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? 1 : 0;
    if (by_box) {
        const EncodeTiledFn enc = encode_tiled();
        if (!enc) return cudaErrorNotSupported;
        cuuint64_t dims[4] = {(cuuint64_t)s.w, (cuuint64_t)s.h, 3, (cuuint64_t)s.n};
        cuuint64_t strides[3] = {(cuuint64_t)s.w * 4, (cuuint64_t)s.w * s.h * 4, (cuuint64_t)s.w * s.h * 12};
        cuuint32_t box[4] = {Tile::RP * 4, Tile::IH, 3, 1}, one[4] = {1, 1, 1, 1};
        if (enc(&image, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(x), dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    const size_t smem = 1024 + Tile::BYTES;
#define OTT_STEMPOOL_LAUNCH(ACT)                                                                                          \
    {                                                                                                                     \
        auto kernel = dense_stem_pool_mma_kernel<S, ACT, OUT8>;                                                           \
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);            \
        if (e != cudaSuccess) return e;                                                                                   \
        e = launch_overlapped(kernel, dim3((unsigned)(blocks < resident ? blocks : resident)), dim3(256), smem, stream, image, x, P, in_scale,  \
                              ep.act_param0, half_bits(ep.rounding), out, s, ph_out, pw_out, tiles_x, tiles_y, (int)blocks,             \
                              make_fast_div((uint32_t)tiles_x), make_fast_div((uint32_t)tiles_y), by_box, pad_zero, status, wait_ns);            \
        if (e != cudaSuccess) return e;                                                                                   \
    }
    switch (ep.act_type) {
        case ACT_RELU: OTT_STEMPOOL_LAUNCH(ACT_RELU) break;
        case ACT_LRELU: OTT_STEMPOOL_LAUNCH(ACT_LRELU) break;
        case ACT_RELU6: OTT_STEMPOOL_LAUNCH(ACT_RELU6) break;
        default: OTT_STEMPOOL_LAUNCH(ACT_NONE) break;
    }
#undef OTT_STEMPOOL_LAUNCH
    return cudaGetLastError();
}

// first layer (fp32 output) + MaxPool 3x3 s2 p1 of its result; out is [n][cout][(oh+1)/2... pooled] fp32 NCHW
cudaError_t launch_dense_stem_pool(cudaStream_t stream, const ConvShape& s, const float* x, const int8_t* w_oihw_host, const float* scale_in_host,
                                   const float* bias_host, const float* scale_out_host, float in_scale, const EpilogueParams& ep, void* out,
                                   int out_dtype, int pad_zero, uint32_t* status, int sm_count, unsigned long long wait_ns) {
    StemParams P{};
    fill_stem_params(P, s, w_oihw_host, scale_in_host, bias_host, out_dtype == DT_S8_NHWC ? scale_out_host : nullptr);
    for (int o = 0; o < ST_COUT_MAX && !ep.has_bias; ++o) P.bias[o] = -0.f;  // (see epilogue.cuh)
    if (out_dtype == DT_S8_NHWC)
        return s.sh == 1 ? launch_pool_s<1, true>(stream, x, P, in_scale, ep, out, s, pad_zero, status, sm_count, wait_ns)
                         : launch_pool_s<2, true>(stream, x, P, in_scale, ep, out, s, pad_zero, status, sm_count, wait_ns);
    return s.sh == 1 ? launch_pool_s<1, false>(stream, x, P, in_scale, ep, out, s, pad_zero, status, sm_count, wait_ns)
                     : launch_pool_s<2, false>(stream, x, P, in_scale, ep, out, s, pad_zero, status, sm_count, wait_ns);
}

// Host-side parameter block: filters OIHW int8 [cout][3][3][3] and the per-channel epilogue vectors.
cudaError_t launch_dense_stem(cudaStream_t stream, const ConvShape& s, const float* x, const int8_t* w_oihw_host, const float* scale_in_host,
                              const float* bias_host, const float* scale_out_host, float in_scale, const EpilogueParams& ep, void* out,
                              int out_dtype) {
    StemParams P{};
    fill_stem_params(P, s, w_oihw_host, scale_in_host, bias_host, scale_out_host);
    if (s.sh == 1) {
        return out_dtype == DT_F32_NCHW ? launch_act<1, DT_F32_NCHW>(stream, x, P, in_scale, ep, out, s)
                                        : launch_act<1, DT_S8_NHWC>(stream, x, P, in_scale, ep, out, s);
    }
    return out_dtype == DT_F32_NCHW ? launch_act<2, DT_F32_NCHW>(stream, x, P, in_scale, ep, out, s)
                                    : launch_act<2, DT_S8_NHWC>(stream, x, P, in_scale, ep, out, s);
}

}  // namespace ottk
