// Depthwise int8 convolution, shared-memory tiled: depthwise_conv2d_int8_x86_pack8_out
// (Tensor/DepthwiseConvKernelInt8X86Pack.cpp:19-119) with the layer's quantize prologue
// (Tensor/QuantizeX86.cpp:396-549) and requantize/dequantize epilogue (Tensor/QuantizeX86.cpp:1723-1870,
// :851-903) fused into one pass over HBM.
//
// One CTA = one image x 32 channels x a band of output rows x up to 64 (stride 2: 40) output columns.
//  1. load: the input halo tile goes to shared memory as int8 *channel planes* (pixels of one channel are
//     consecutive bytes). From fp32 NCHW it is quantized on the way: a thread takes one 4-pixel word position of eight
//     channels, so that the position's index arithmetic and bounds tests are paid once per eight words and eight 16-byte loads
//     are in flight per thread. Words start on 16-byte boundaries of the tensor whatever the width is; a row's first pixel
//     then lies `sh` (0..3) bytes into its first word, and the compute phase shifts each row by its own amount. From int8
//     NHWC the 16-byte channel vectors of 4 neighbouring pixels are transposed in registers (4x4 byte transposes).
//  2. compute: thread = (channel = lane, 4 consecutive output columns), walking down the band. Because pixels are consecutive bytes, one 32-bit window holds 4 horizontal taps of one channel and a dp4a does 4 multiply-adds; the
//     windows of the last K input rows stay in registers while the thread walks down its rows. The fifth column of a 5x5
//     filter would waste three quarters of a dp4a per row, so its bytes are collected down the column instead (one byte
//     permute per row): 7 dp4a per output instead of 10. Sums are exact s32.
//  3. epilogue in registers (epilogue.cuh). int8 results: a 4x4 byte transpose across four lanes (two shuffles) gives every
//     lane four channels of one pixel; eight lanes write a pixel's 32 channels, one whole sector. fp32 NCHW results are
//     stored directly. No staging buffer and no second barrier: warps leave one by one, and more CTAs fit an SM.
// Bound by instruction issue on large fp32 inputs (the quantizer alone is 4 instructions per element) and by latency on small
// maps, where the plan cuts the band and the rows per thread until the GPU has about two CTAs per SM.
//
// This header holds the kernel template; depthwise_tiled_k*s*.cu instantiate it per (kernel size, stride)
// so the variants compile in parallel.
#pragma once

#include <mutex>
#include <type_traits>

#include "launch.cuh"
#include "store.cuh"

namespace ottk {
namespace dwt {

constexpr int CG = 32;  // channels per CTA: eight lanes of four channels
constexpr int THREADS = 256;
constexpr int LOAD_CH = 8;              // channels per load item (fp32 input)
enum : int { EPI_S8 = 0, EPI_F32 = 1 };

struct Tile {
    int ty, nxq;          // output rows / groups of 4 output columns per CTA
    int nrg, rpt;         // row groups per CTA and rows of one group (= per thread)
    int ir, rp, ps;       // input tile: rows, row pitch and plane stride in 32-bit words (ps odd)
    int tiles_y, tiles_x, cgroups;
    int threads;
    uint32_t div_rp, div_nxq;  // ceil(2^20 / x): exact quotients for the small indices they are used on
};

template <int K, int S>
struct Geo {
    static constexpr int KK = (K + 3) / 4;           // packed filter words per filter row
    static constexpr int NRAW = S == 1 ? 3 : 4;      // aligned words under a thread's 4 outputs, in one input row
};

// The last K input rows under the thread's 4 outputs, as windows in registers: win[slot][t] = bytes [t*S, +4) of the row counted
// from the first input column of output 0 (slot = input row % K), and for K = 5 the fifth column's bytes of the last four rows.
template <int K, int S>
struct RowRing {
    static constexpr int NAL = Geo<K, S>::NRAW - 1;
    uint32_t win[K][4], vert[4], al[NAL];
    static __device__ __forceinline__ constexpr int tail_word(int t) { return S == 1 ? 1 : 1 + (t >> 1); }
    static __device__ __forceinline__ constexpr int tail_byte(int t) { return S == 1 ? t : 2 * (t & 1); }

    // `sh` = 8 * the byte offset of output 0's first column inside its aligned word (modulo 32)
    __device__ __forceinline__ void load(uint32_t (&w)[4], const uint32_t* __restrict__ p, int sh) {
        uint32_t raw[NAL + 1];
#pragma unroll
        for (int i = 0; i < NAL + 1; ++i) raw[i] = p[i];
#pragma unroll
        for (int i = 0; i < NAL; ++i) al[i] = __funnelshift_r(raw[i], raw[i + 1], sh);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const int wi = (t * S) >> 2, bs = ((t * S) & 3) * 8;  // compile-time after unrolling
            w[t] = bs == 0 ? al[wi] : __funnelshift_r(al[wi], al[wi + 1], bs);
        }
    }
    // the fifth column, oldest row in byte 0: drop the oldest row, append the row last loaded
    __device__ __forceinline__ void push_tail() {
#pragma unroll
        for (int t = 0; t < 4; ++t) vert[t] = __byte_perm(vert[t], al[tail_word(t)], 0x0321 | ((4 + tail_byte(t)) << 12));
    }
    __device__ __forceinline__ void prime(int r, const uint32_t* __restrict__ p, int sh) {
        load(win[r % K], p, sh);
        if (K == 5) {
            if (r == 0) vert[0] = vert[1] = vert[2] = vert[3] = 0u;
            push_tail();
        }
    }
    // Loads the S rows that output row R (mod K) needs beyond those of the row before it and multiplies.
    template <int R>
    __device__ __forceinline__ void advance(const uint32_t* __restrict__& p, int rp, int& sh, int wmod8, const uint32_t (&wk)[K], uint32_t wv,
                                            uint32_t w44, int (&acc)[4]) {
        constexpr int base = (R * S) % K;
#pragma unroll
        for (int ky = K - S; ky < K; ++ky) {
            if (K == 5 && ky > K - S) push_tail();  // (stride 2: the first of the two new rows)
            load(win[(base + ky) % K], p, sh);
            p += rp;
            sh += wmod8;
        }
#pragma unroll
        for (int ky = 0; ky < K; ++ky)
#pragma unroll
            for (int t = 0; t < 4; ++t) acc[t] = __dp4a((int)win[(base + ky) % K][t], (int)wk[ky], acc[t]);
        if (K == 5) {
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                acc[t] = __dp4a((int)vert[t], (int)wv, acc[t]);
                acc[t] = __dp4a((int)al[tail_word(t)], (int)(w44 << (8 * tail_byte(t))), acc[t]);
            }
            push_tail();
        }
    }
};

// Added to the activation (ReLU, ReLU6) of an int8 build: EpilogueParams::signed_rounding. (ReLU is not the LeakyReLU of slope 0: a bias of
// -infinity, a channel that is switched off, would become a NaN.)
constexpr int kSignedRounding = 8;

// Four accumulators of one channel -> four int8 in one word, the arithmetic as packed pairs.
// LONG: the constant of the fused product and sum takes the sum's sign, which is + (or that of a -0, and the result 0 all the same), in one value of
// each pair. That instruction makes the compiler keep 80 registers where it makes do with 71, and the latency of a band, which bounds the
// smaller launches, is shorter. For the one instance that had 80 before its rounding was mended (5x5, ReLU6; us with 71 / this / two
// roundings: 96 channels 40x40 x32 9.92 / 7.93 / 8.27, 75 66x15 x25 5.55 / 4.99 / 5.20, x100 13.2 / 13.7 / 14.4, 96 40x40 x128 24.8 / 27.3 / 29.3).
template <int ACT, bool SIGNED, bool LONG>
__device__ __forceinline__ uint32_t epi_s8x4(const int (&acc)[4], float si, float bi, float so, float p0, uint32_t half) {
    const float2 s2 = make_float2(si, si), b2 = make_float2(bi, bi), o2 = make_float2(so, so);
    int2 q[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float2 v = __ffma2_rn(make_float2(__int2float_rn(acc[2 * h]), __int2float_rn(acc[2 * h + 1])), s2, b2);
        const float2 y = make_float2(activate_t<ACT>(v.x, p0), activate_t<ACT>(v.y, p0));
        if (LONG) {
            const float2 r = __ffma2_rn(y, o2, make_float2(half_signed(y.x, kHalfFused), __uint_as_float(kHalfFused)));
            q[h] = make_int2(__float2int_rz(r.x), __float2int_rz(r.y));
        } else {
            q[h] = round2_act<ACT, SIGNED>(y, o2, half);
        }
    }
    return pack_sat_s8x4(q[0].x, q[0].y, q[1].x, q[1].y);
}

template <int K, int S, bool IN_F32, int EPI, int ACT_BUILD>
__global__ void __launch_bounds__(THREADS, K == 3 ? 4 : 3)
depthwise_tiled_kernel(const void* __restrict__ xin, const __grid_constant__ PlaneGather G, const uint32_t* __restrict__ wq,
                       const float* __restrict__ in_scales, int n_in_scales, EpilogueParams ep, void* __restrict__ out, ConvShape s, Tile T,
                       int aligned) {
    constexpr int KK = Geo<K, S>::KK, ACT = ACT_BUILD & ~kSignedRounding;
    constexpr bool SIGNED = (ACT_BUILD & kSignedRounding) != 0;
    constexpr bool LONG = K == 5 && S == 1 && !IN_F32 && EPI == EPI_S8 && ACT_BUILD == ACT_RELU6;
    extern __shared__ uint32_t smem[];
    __shared__ const float* ch_ptr[CG];
    __shared__ float ch_scale[CG];
    pdl_launch_dependents();
    uint32_t* tin = smem;  // [32][ir][rp] (+pad): int8 channel planes of the input tile

    int b = blockIdx.x;
    const int cg = b % T.cgroups; b /= T.cgroups;
    const int tx = b % T.tiles_x; b /= T.tiles_x;
    const int tyi = b % T.tiles_y;
    const int img = b / T.tiles_y;
    const int c0 = cg * CG;
    const int oy0 = tyi * T.ty, ox0 = tx * T.nxq * 4;
    const int iy0 = oy0 * S - s.ph;
    const int ix_first = ox0 * S - s.pw;  // first input column the tile needs
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = (int)blockDim.x >> 5;

    // the lane's channel: filter and epilogue constants (they do not depend on the previous kernel)
    const int c = c0 + lane;
    const bool c_ok = c < s.cout_pad;
    uint32_t wk[K], wv = 0u, w44 = 0u;  // filter rows, first four columns; the fifth column's first four rows; its last row
    {
        uint32_t wd[K * KK];
#pragma unroll
        for (int i = 0; i < K * KK; ++i) wd[i] = c_ok ? __ldg(wq + (long)c * K * KK + i) : 0u;
#pragma unroll
        for (int ky = 0; ky < K; ++ky) wk[ky] = wd[ky * KK];
        if (K == 5) {
            wv = __byte_perm(__byte_perm(wd[1], wd[3], 0x0040), __byte_perm(wd[5], wd[7], 0x0040), 0x5410);
            w44 = wd[9];
        }
    }
    const float p_si = c_ok ? __ldg(ep.scale_in + c) : 0.f;
    const float p_bi = c_ok ? bias_or_neutral(ep, c) : 0.f;
    const uint32_t half = half_bits(ep.rounding);
    const float p_so = c_ok && EPI != EPI_F32 ? __ldg(ep.scale_out + c) : 0.f;
    if (IN_F32 && tid < CG && c0 + tid < s.cin) {
        ch_ptr[tid] = G.plane(c0 + tid, img, (long)s.h * s.w);
        ch_scale[tid] = n_in_scales == 1 ? __ldg(in_scales) : __ldg(in_scales + c0 + tid);
    }
    if (IN_F32) __syncthreads();
    pdl_wait();

    // ---- 1. load the input tile ----
    const int npos = T.ir * T.rp;
    const int wmod = IN_F32 && !aligned ? s.w & 3 : 0;  // how the byte offset of a row's first pixel moves from row to row
    if (IN_F32) {
        const int chunks = (min(CG, s.cin - c0) + LOAD_CH - 1) / LOAD_CH;
        for (int i = tid, chunk = 0; ; i += (int)blockDim.x) {
            while (i >= npos) { i -= npos; ++chunk; }
            if (chunk >= chunks) break;
            const int r = (int)(((uint32_t)i * T.div_rp) >> 20), xw = i - r * T.rp;
            const int iy = iy0 + r, cl0 = chunk * LOAD_CH;
            const bool row_ok = iy >= 0 && iy < s.h;
            // (the planes past the last channel of an incomplete chunk repeat its last one: their filters are zero)
            const int cl_last = min(CG, s.cin - c0) - 1;
            uint32_t* dst = tin + cl0 * T.ps + i;
            if (aligned) {
                // every 16-byte word lies wholly inside the row or wholly outside
                const int ix = (ix_first & ~3) + xw * 4;
                if (row_ok && ix >= 0 && ix < s.w) {
                    const int off = iy * s.w + ix;
                    float4 v[LOAD_CH];
#pragma unroll
                    for (int k = 0; k < LOAD_CH; ++k) v[k] = __ldg(reinterpret_cast<const float4*>(ch_ptr[min(cl0 + k, cl_last)] + off));
#pragma unroll
                    for (int k = 0; k < LOAD_CH; ++k) dst[k * T.ps] = quantize4_pack(v[k].x, v[k].y, v[k].z, v[k].w, ch_scale[min(cl0 + k, cl_last)], half);
                } else {
#pragma unroll
                    for (int k = 0; k < LOAD_CH; ++k) dst[k * T.ps] = 0u;
                }
            } else {
                // the word that starts on a 16-byte boundary of the tensor: whole words inside the row are one load, words that
                // reach over a row's end take their pixels one by one
                float4 v[LOAD_CH];
#pragma unroll
                for (int k = 0; k < LOAD_CH; ++k) {
                    v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row_ok) {
                        const float* row = ch_ptr[min(cl0 + k, cl_last)] + iy * s.w;
                        const int sh = ((int)(reinterpret_cast<uintptr_t>(row) >> 2) + ix_first) & 3;
                        const int ix = ix_first - sh + xw * 4;
                        if (ix >= 0 && ix + 3 < s.w) {
                            v[k] = __ldg(reinterpret_cast<const float4*>(row + ix));
                        } else {
                            if (ix >= 0 && ix < s.w) v[k].x = __ldg(row + ix);
                            if (ix + 1 >= 0 && ix + 1 < s.w) v[k].y = __ldg(row + ix + 1);
                            if (ix + 2 >= 0 && ix + 2 < s.w) v[k].z = __ldg(row + ix + 2);
                            if (ix + 3 >= 0 && ix + 3 < s.w) v[k].w = __ldg(row + ix + 3);
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < LOAD_CH; ++k) dst[k * T.ps] = quantize4_pack(v[k].x, v[k].y, v[k].z, v[k].w, ch_scale[min(cl0 + k, cl_last)], half);
            }
        }
    } else {
        // Each 16-channel group is read from one tensor: the layer's own input, or (a layer created with gathered input)
        // 16 channels of one of several source tensors, named by the table: ref = (tensor << 24) | first channel, and
        // img_stride[tensor] = that tensor's channel stride.
        const int half = tid & 1;  // blockDim.x is even: a thread stays on its half
        const int ch = c0 + half * 16;
        const int8_t* x = static_cast<const int8_t*>(xin) + (long)img * s.h * s.w * s.cin_pad + ch;
        long pitch = s.cin_pad;
        if (G.base[0] != nullptr && ch < s.cin_pad) {
            const uint32_t ref = G.ref[ch >> 4];
            pitch = (long)G.img_stride[ref >> 24];
            x = reinterpret_cast<const int8_t*>(G.base[ref >> 24]) + (long)img * s.h * s.w * pitch + (ref & 0xFFFFFFu);
        }
        if (ch < s.cin_pad) {
            for (int i = tid >> 1; i < npos; i += (int)blockDim.x >> 1) {  // one pixel quad
                const int r = (int)(((uint32_t)i * T.div_rp) >> 20), xw = i - r * T.rp;
                const int iy = iy0 + r, ix = (ix_first & ~3) + xw * 4;
                const bool row_ok = iy >= 0 && iy < s.h;
                uint4 v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[j] = make_uint4(0, 0, 0, 0);
                    if (row_ok && ix + j >= 0 && ix + j < s.w) v[j] = __ldg(reinterpret_cast<const uint4*>(x + ((long)iy * s.w + ix + j) * pitch));
                }
                uint32_t* dst = tin + (half * 16) * T.ps + i;
                uint32_t o[4];
                transpose4x4(v[0].x, v[1].x, v[2].x, v[3].x, o);
#pragma unroll
                for (int k = 0; k < 4; ++k) dst[(0 + k) * T.ps] = o[k];
                transpose4x4(v[0].y, v[1].y, v[2].y, v[3].y, o);
#pragma unroll
                for (int k = 0; k < 4; ++k) dst[(4 + k) * T.ps] = o[k];
                transpose4x4(v[0].z, v[1].z, v[2].z, v[3].z, o);
#pragma unroll
                for (int k = 0; k < 4; ++k) dst[(8 + k) * T.ps] = o[k];
                transpose4x4(v[0].w, v[1].w, v[2].w, v[3].w, o);
#pragma unroll
                for (int k = 0; k < 4; ++k) dst[(12 + k) * T.ps] = o[k];
            }
        }
    }
    __syncthreads();

    // ---- 2. compute + 3. epilogue ----
    const int rows_out = min(T.ty, s.oh - oy0);
    const long oplane = (long)s.oh * s.ow;
    const uint32_t* plane = tin + lane * T.ps;
    // byte offset of the tile's first input column in its first aligned word, times 8; row r's is wmod8 * r further (mod 32: the
    // funnel shifts take their amount modulo 32)
    int sh8 = ix_first * 8;
    if (IN_F32 && !aligned && c < s.cin) sh8 += ((int)(reinterpret_cast<uintptr_t>(ch_ptr[lane]) >> 2) + iy0 * wmod) * 8;
    const int wmod8 = wmod * 8;
    // int8 output: after the exchange below lane 4k + p holds pixel p's channels 4k .. 4k + 3
    const int px = lane & 3, cq = c0 + (lane & ~3);
    const uint32_t sel_a = px < 2 ? 0x5410u : 0x3276u, sel_b = (px & 1) == 0 ? 0x6240u : 0x3715u;
    for (int item = warp; item < T.nxq * T.nrg; item += nwarps) {
        const int rg = (int)(((uint32_t)item * T.div_nxq) >> 20), xq = item - rg * T.nxq;
        const int ox = ox0 + xq * 4, r0 = rg * T.rpt;
        const int nrows = min(T.rpt, rows_out - r0);
        if (ox >= s.ow || nrows <= 0) continue;  // warp-uniform
        RowRing<K, S> ring;
        const uint32_t* p = plane + r0 * S * T.rp + xq * S;
        int sh = sh8 + r0 * S * wmod8;
#pragma unroll
        for (int r = 0; r < K - S; ++r) {
            ring.prime(r, p, sh);
            p += T.rp;
            sh += wmod8;
        }
        int8_t* o8 = nullptr;
        float* of = nullptr;
        bool store_ok;
        if (EPI == EPI_F32) {
            of = reinterpret_cast<float*>(out) + ((long)img * s.cout + c) * oplane + (long)(oy0 + r0) * s.ow + ox;
            store_ok = c < s.cout;
        } else {
            o8 = reinterpret_cast<int8_t*>(out) + (((long)img * s.oh + oy0 + r0) * s.ow + ox + px) * s.cout_pad + cq;
            store_ok = ox + px < s.ow && cq < s.cout_pad;
        }
        const int ow_left = s.ow - ox;
        const long row_step = EPI == EPI_F32 ? (long)s.ow : (long)s.ow * s.cout_pad;
        auto step = [&](auto rc) {
            constexpr int R = decltype(rc)::value;  // output row modulo K: fixes the ring slots at compile time
            int acc[4] = {0, 0, 0, 0};
            ring.template advance<R>(p, T.rp, sh, wmod8, wk, wv, w44, acc);
            if (EPI != EPI_F32) {
                uint32_t w = epi_s8x4<ACT, SIGNED, LONG>(acc, p_si, p_bi, p_so, ep.act_param0, half);
                w = __byte_perm(w, __shfl_xor_sync(0xFFFFFFFFu, w, 2), sel_a);
                w = __byte_perm(w, __shfl_xor_sync(0xFFFFFFFFu, w, 1), sel_b);
                if (store_ok) *reinterpret_cast<uint32_t*>(o8) = w;
                o8 += row_step;
            } else {
                float v[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) v[t] = activate_t<ACT>(__fmaf_rn(__int2float_rn(acc[t]), p_si, p_bi), ep.act_param0);
                if (store_ok) {
                    if (ow_left >= 4 && (reinterpret_cast<uintptr_t>(of) & 15) == 0) {
                        *reinterpret_cast<float4*>(of) = make_float4(v[0], v[1], v[2], v[3]);
                    } else {
#pragma unroll
                        for (int t = 0; t < 4; ++t)
                            if (t < ow_left) of[t] = v[t];
                    }
                }
                of += row_step;
            }
        };
        for (int oy = 0; oy < nrows; oy += K) {
            step(std::integral_constant<int, 0>{});
            if (oy + 1 < nrows) step(std::integral_constant<int, 1>{});
            if (oy + 2 < nrows) step(std::integral_constant<int, 2>{});
            if (K > 3) {
                if (oy + 3 < nrows) step(std::integral_constant<int, 3>{});
                if (oy + 4 < nrows) step(std::integral_constant<int, 4>{});
            }
        }
    }
}

// Tile of a layer. Columns: equal tiles of at most 64 (stride 2: 40) outputs. Warps share the (column group, row group) items.
// Rows: bands of equal height, as many rows as a channel plane of kPlaneWords words holds at most. Which number of bands is
// best depends on how the CTAs fall on the SMs, so each is rated by the larger of what bounds it: the instructions of the SM with most CTAs (about 2.5 per cycle are
// issued), or the latency of one CTA (memory round trip, then one warp's dependent instructions at six cycles each) times the
// waves. The instruction counts are those of the inner loops: 26 per fp32 word loaded and quantized, 7 per 32 int8 quads
// loaded and transposed, 46 / 75 per warp and output row of a 3x3 / 5x5 filter, 12 per row that only fills the ring. Counting the warps that
// have no item in the last pass as if they issued kept eight-warp CTAs from launches that want them: 3x3 256 channels fp32 -> int8 56x56
// x64 68.6 -> 65.7 us; fp32 -> fp32 from 15 us on 1.09 times as fast, the rest of 360 layers 0.99 to 1.03. Low bands (below) are counted
// that way all the same: what bounds them is the stores, and a count without idle warps picks bands that leave many of them (236 channels 57x72 x45 100 us, 74.9 this way;
// 261 35x11 x78 37.6 / 33.4; 130 such layers on average the same).
// fp32 output from int8, stride 1: a lane stores 16 bytes of its own channel's plane, half a sector (single pixels where the rows are not
// aligned), and the rest of the sector and of the line comes from the next warps. An output that does not fit L2, or one of single
// pixels, wants that to happen soon: low bands (planes of 128 words), eight warps side by side on the same rows. us, high bands / low:
// 5x5 256 channels 56x56 x64 194 / 114, 116 30x73 x110 182 / 110, 288 15x9 x71 20.1 / 15.4; 3x3 251 67x33 x52 195 / 117. But 5x5 199
// 25x56 x69, 77 MB of aligned rows, 34.7 / 38.7.
constexpr int kPlaneWords = 384, kLowPlaneWords = 128, kSms = 148;
constexpr long kBeyondL2 = 96l << 20, kMuchOutput = 8l << 20;
template <int K, int S, bool IN_F32, int EPI>
inline Tile plan_tile(const ConvShape& s) {
    Tile T{};
    const bool low = !IN_F32 && EPI == EPI_F32 && S == 1 && 4l * s.n * s.cout * s.oh * s.ow >= (s.ow % 4 == 0 ? kBeyondL2 : kMuchOutput);
    const int ow4 = (s.ow + 3) / 4, max_nxq = S == 1 ? 16 : 10;
    T.tiles_x = (ow4 + max_nxq - 1) / max_nxq;
    T.nxq = (ow4 + T.tiles_x - 1) / T.tiles_x;
    T.rp = (T.nxq - 1) * S + Geo<K, S>::NRAW;
    T.cgroups = (s.cout_pad + CG - 1) / CG;
    const int ty_max = ((low ? kLowPlaneWords : kPlaneWords) / T.rp - K) / S + 1;
    const long per_band = (long)s.n * T.tiles_x * T.cgroups;
    // a throughput-bound launch wants every warp to have the same work, a latency-bound one as many warps as there are
    // (fp32 input: of two that are rated alike the wider one, which has more loads under way)
    const int few = low ? THREADS / 32 : T.nxq > 8 ? (T.nxq + 1) / 2 : T.nxq > 2 ? T.nxq : 2;
    const int widths[2] = {IN_F32 ? THREADS / 32 : few, IN_F32 ? few : THREADS / 32};
    double best = 0;
    for (int bands = (s.oh + ty_max - 1) / ty_max; bands <= s.oh; ++bands) {
        const int ty = (s.oh + bands - 1) / bands, tiles_y = (s.oh + ty - 1) / ty;
        if (tiles_y < bands) continue;  // no band is lower than with fewer of them
        const long ctas = per_band * tiles_y;
        const int npos = ((ty - 1) * S + K) * T.rp;
        for (int w : widths) {
            int nrg = 1;
            while ((!low || T.nxq <= 2) && T.nxq * nrg < w && ty > 2 * nrg) ++nrg;
            const int rpt = (ty + nrg - 1) / nrg;
            nrg = (ty + rpt - 1) / rpt;
            const int passes = (T.nxq * nrg + w - 1) / w;
            const double load = npos * (IN_F32 ? 26.0 : 7.0), item = rpt * (K == 3 ? 46.0 : 75.0) + (K - S) * 12.0;
            const double instr = load + passes * w * item, issued = low ? instr : load + T.nxq * nrg * item;  // (a warp without an item in the last pass issues nothing)
            int resident = 65536 / ((K == 3 ? 64 : 80) * 32 * w);
            const int by_smem = 224 * 1024 / (CG * 4 * npos + 2048);
            if (by_smem < resident) resident = by_smem;
            const double waves = (double)ctas / ((double)kSms * resident);
            const double busy = (double)((ctas + kSms - 1) / kSms) * issued / 2.5;
            const double chain = (waves <= 1.0 ? 1.0 : waves + 0.5) * (1800.0 + 6.0 * instr / w);
            const double score = busy > chain ? busy : chain;
            if (T.ty != 0 && score >= best) continue;
            best = score;
            T.ty = ty; T.tiles_y = tiles_y; T.nrg = nrg; T.rpt = rpt; T.threads = 32 * w;
        }
        if (ty <= 2) break;
    }
    T.ir = (T.ty - 1) * S + K;
    T.ps = T.ir * T.rp;
    if (T.ps % 2 == 0) T.ps += 1;
    T.div_rp = ((1u << 20) + T.rp - 1) / T.rp;
    T.div_nxq = ((1u << 20) + T.nxq - 1) / T.nxq;
    return T;
}

template <int K, int S, bool IN_F32, int EPI, int ACT>
cudaError_t launch_t(cudaStream_t stream, const ConvShape& s, const void* x, const PlaneGather& G, const uint32_t* wq, const float* in_scales,
                     int n_in_scales, const EpilogueParams& ep, void* out) {
    const Tile T = plan_tile<K, S, IN_F32, EPI>(s);
    const size_t smem = (size_t)CG * T.ps * 4;
    // fp32 rows whose 16-byte words never cross a row's end: a width that is a multiple of 4 and 16-byte aligned planes
    int aligned = s.w % 4 == 0 ? 1 : 0;
    for (int i = 0, last = -1; IN_F32 && i < s.cin && aligned; ++i) {
        const int b = (int)(G.ref[i] >> 24);
        if (b != last && ((reinterpret_cast<uintptr_t>(G.base[b]) & 15) != 0 || G.img_stride[b] % 4 != 0)) aligned = 0;
        last = b;
    }
    auto kernel = depthwise_tiled_kernel<K, S, IN_F32, EPI, ACT>;
    static std::mutex mu;  // several host threads may drive different GPUs through this function at once
    static bool attr_set[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) {
        std::lock_guard<std::mutex> lock(mu);
        if (!attr_set[dev]) {
            cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
            if (e != cudaSuccess) return e;
            attr_set[dev] = true;
        }
    }
    const long blocks = (long)s.n * T.tiles_y * T.tiles_x * T.cgroups;
    if (blocks == 0) return cudaSuccess;
    return launch_overlapped(kernel, dim3((unsigned)blocks), dim3(T.threads), smem, stream, x, G, wq, in_scales, n_in_scales, ep, out, s, T, aligned);
}

template <int K, int S, bool IN_F32, int EPI>
cudaError_t launch_act(cudaStream_t stream, const ConvShape& s, const void* x, const PlaneGather& G, const uint32_t* wq, const float* in_scales,
                       int n_in_scales, const EpilogueParams& ep, void* out) {
    if constexpr (EPI != EPI_F32) {
        if (ep.signed_rounding && ep.act_type == ACT_RELU)
            return launch_t<K, S, IN_F32, EPI, ACT_RELU | kSignedRounding>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
        if (ep.signed_rounding && ep.act_type == ACT_RELU6)
            return launch_t<K, S, IN_F32, EPI, ACT_RELU6 | kSignedRounding>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
    }
    switch (ep.act_type) {
        case ACT_RELU: return launch_t<K, S, IN_F32, EPI, ACT_RELU>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
        case ACT_LRELU: return launch_t<K, S, IN_F32, EPI, ACT_LRELU>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
        case ACT_RELU6: return launch_t<K, S, IN_F32, EPI, ACT_RELU6>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
        default: return launch_t<K, S, IN_F32, EPI, ACT_NONE>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
    }
}

template <int K, int S>
cudaError_t launch_ks(cudaStream_t stream, const ConvShape& s, const void* x, const PlaneGather& G, int in_dtype, const uint32_t* wq,
                      const float* in_scales, int n_in_scales, const EpilogueParams& ep, void* out, int out_dtype) {
    const bool f32in = in_dtype == DT_F32_NCHW;
    if (out_dtype == DT_F32_NCHW)
        return f32in ? launch_act<K, S, true, EPI_F32>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out)
                     : launch_act<K, S, false, EPI_F32>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
    return f32in ? launch_act<K, S, true, EPI_S8>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out)
                 : launch_act<K, S, false, EPI_S8>(stream, s, x, G, wq, in_scales, n_in_scales, ep, out);
}

}  // namespace dwt

// defined one per file (depthwise_tiled_k3s1.cu ...)
cudaError_t launch_depthwise_tiled_k3s1(cudaStream_t, const ConvShape&, const void*, const PlaneGather&, int, const uint32_t*, const float*, int, const EpilogueParams&, void*, int);
cudaError_t launch_depthwise_tiled_k3s2(cudaStream_t, const ConvShape&, const void*, const PlaneGather&, int, const uint32_t*, const float*, int, const EpilogueParams&, void*, int);
cudaError_t launch_depthwise_tiled_k5s1(cudaStream_t, const ConvShape&, const void*, const PlaneGather&, int, const uint32_t*, const float*, int, const EpilogueParams&, void*, int);
cudaError_t launch_depthwise_tiled_k5s2(cudaStream_t, const ConvShape&, const void*, const PlaneGather&, int, const uint32_t*, const float*, int, const EpilogueParams&, void*, int);

}  // namespace ottk
