// Dense int8 convolution as an implicit GEMM on the sm_100a tensor cores.
//
// Replaces the reference's im2col + sgemm int8 path (Tensor/ConvolutionMM2DInt8X86Pack.cpp:2369-2445 builds
// the im2col matrix, :1656-2223 is the s8 x s8 -> s32 GEMM, :2533-2556 the 1x1 shortcut) and the epilogue
// passes that follow it (Tensor/QuantizeX86.cpp:851-903 dequantize, :1723-1870 requantize). No im2col
// matrix, no s32 tensor and no padded copy ever reach HBM:
//
//   D[128 pixels, BN out-channels] (s32, in TMEM)  +=  A[128 pixels, 32..128 in-channels] * B[BN, same]^T
//
// * A tiles come straight from the NHWC int8 activations with 4-D TMA boxes {channels, TW, TH, 1};
//   out-of-image rows/columns are zero-filled by TMA, which is the reference's constant_pad
//   (Tensor/Padding.cpp:22-36). 1x1 convolutions view the activations as a flat [pixels, channels] matrix so
//   tiles never straddle anything. k x k convolutions load, per pixel tile of 8 x 16 and channel block, ONE box
//   that holds the tile and its halo; filter tap (ky, kx) is an MMA whose A descriptor starts (ky, kx) pixels
//   into that box and steps one halo row per 8-row group (the swizzle is a function of the shared-memory
//   address, so shifted views read what TMA wrote). At stride 2 there are two boxes, one per column parity, where the
//   map suits them (umma_prefers_parity); other strides and dilated layers load one shifted box per tap instead.
// * B (the layer's weights for this CTA's BN output channels, all taps) is loaded once per CTA and stays in
//   shared memory while the CTA walks over its pixel tiles (persistent, weight-stationary).
// * tcgen05.mma.kind::i8 accumulates exact s32 in TMEM; two accumulators (four of at most 64 columns; one in a
//   compact launch) let the epilogue of tile i overlap the loads and MMAs of the tiles behind it.
// * The epilogue warps read TMEM (tcgen05.ld), apply fma(acc, scale_in, bias) -> activation -> requantize
//   (epilogue.cuh) and store int8 NHWC / fp32 NCHW / s32 NHWC.
// * Long 1x1 launches with int8 output exchange the operands, D[128 channels, pixels], see the comment on the builds in front of the kernel.
//
// Warp roles (320 threads): warp 0 = TMA producer (one elected thread), warp 1 = TMEM owner + MMA issuer (one elected thread),
// warps 2..9 = epilogue: warp w reads TMEM lanes 32*(w%4)..+31 (the hardware's lane window of a warp) and
// shares that quarter's column chunks with the other warps of the same window, dealt out over all the CTA's tiles.
// Every mbarrier wait is bounded in time: on expiry the waiter raises a CTA-wide abort flag, ORs a code
// into the status word, and all roles fall through to the common teardown, which frees TMEM.
#include <cuda.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "dense_umma.h"
#include "launch.cuh"
#include "umma_primitives.cuh"

namespace ottk {

namespace {

constexpr int kMaxEpiWarps = 8;                     // 2 per TMEM lane quarter
constexpr int kMaxThreads = 64 + 32 * kMaxEpiWarps;  // UmmaPlan::epi_warps is 4 or 8 (16 in the wide-tile build)
constexpr int kTileM = 128;
constexpr int kMaxAccBufs = 8;
constexpr uint32_t kHalfSm = 113 * 1024;  // shared memory of a CTA that leaves room for another like it
constexpr int kHaloTw = 8, kHaloTh = 16;  // pixel tile of the halo mode: 8 wide so that a tile row is one 8-row operand group
using namespace umma;

// Activation tensor maps of one launch: one for an ordinary layer; one per source tensor for a layer whose K blocks are
// gathered from several int8 tensors.
struct KernelMaps {
    CUtensorMap tm[kUmmaMaxSources];
    uint16_t block_x[kUmmaMaxGatherBlocks];
    uint8_t block_src[kUmmaMaxGatherBlocks];
};

// Added to the activation of an int8 build: scale_out is one scalar. The parameters are what the epilogue waits for (a float4 from
// shared memory, the same for all lanes, takes two passes of the data pipe that the output stores need too): a third fewer of
// them, 64 -> 256 56x56 x128 without activation 51.9 -> 48.1 us. A test inside one build costs as much as it saves.
constexpr int kOneScale = 8;
// Compact builds: the output kind and the activation are arguments and nothing large is unrolled, so that every layer of a network's
// small launches runs the same 39 KB of code. A specialised build is 60 to 110 KB, of which a launch runs about a third; when the
// launch before it ran another build, its instructions come from L2 again: 20x20x116 -> 116, one image, us per launch, specialised /
// compact: the same layer over and over 2.57 / 2.65, two activations in turn 3.20 / 2.63, five builds in turn 4.07 / 2.63.
constexpr int kAnyOut = 7, kAnyAct = 7;
constexpr int kCompactBuild = 4, kCompactQuantBuild = 5;
// Builds whose accumulator rows are output channels (int8 output): see UmmaPlan::rows. Two CTAs per SM, one with sixteen epilogue warps, or
// one that quantizes fp32 input.
constexpr int kRowsBuild = 6, kRowsWideBuild = 7, kRowsQuantBuild = 8;
constexpr __host__ __device__ bool build_rows(int build) { return build == kRowsBuild || build == kRowsWideBuild || build == kRowsQuantBuild; }
constexpr __host__ __device__ bool build_quantizes(int build) { return build == 3 || build == kCompactQuantBuild || build == kRowsQuantBuild; }
constexpr int kQuantBuild = 3, kQuantWarps = 8, kQuantRuns = 2;
constexpr int kOutSlots = 4;  // finished tiles on their way out, at most
// pixels (accumulator columns) of a tile, and epilogue warps that share an accumulator: 64 of either's results per thread
constexpr __host__ __device__ int rows_pixels(int build) { return build == kRowsQuantBuild ? 64 : 128; }
constexpr __host__ __device__ int team_warps(int build) { return rows_pixels(build) / 16; }
constexpr int kRowsMaxBlocks = 4;
// kRowsQuantBuild: quantizing warps, and the boxes of fp32 planes that they read, 16 channels x 64 pixels each
constexpr int kBoxWarps = 10, kBoxChannels = 16;
constexpr uint32_t kBoxBytes = 4096;
constexpr __host__ __device__ int build_threads(int build) {
    return build == kRowsQuantBuild ? 96 + 32 * (8 + kBoxWarps) : build == kRowsWideBuild ? 96 + 32 * 16 : build == kRowsBuild ? 96 + 32 * 8 : build == 2 || build_quantizes(build) ? 64 + 32 * 16 : kMaxThreads;
}

// fp32 input of a launch that quantizes on the way in (kQuantBuild)
struct QuantSource {
    // the input's channels as at most kQuantRuns runs of consecutive planes of a tensor (a Concat of two blobs is two runs):
    // run i starts at channel first[i], whose plane is at base[i]; unused runs start past the last channel
    const float* base[kQuantRuns];
    long long img_stride[kQuantRuns];
    int first[kQuantRuns];
    float scale;
    uint32_t half;           // rounding constant
    int vec;                 // rows of four pixels are whole and 16-byte aligned
    FastDiv div_halo;        // by the width of a halo tile
    __device__ __forceinline__ const float* plane(int c, int img, int hw) const {
        const int i = c >= first[1] ? 1 : 0;
        return base[i] + (long long)img * img_stride[i] + (long long)(c - first[i]) * hw;
    }
};

// Address of 16-byte chunk `chunk` of row `row` of an operand tile of bkc-byte rows at `tile` (1 KiB aligned): the swizzle TMA
// applies for this row width.
__device__ __forceinline__ uint32_t operand_chunk(uint32_t tile, int bkc, int row, int chunk) {
    const uint32_t a = tile + (uint32_t)(row * bkc + chunk * 16);
    return a ^ (((a >> 7) & ((uint32_t)(bkc >> 4) - 1u)) << 4);
}

__device__ __forceinline__ void store_chunk(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// The same position of 16 channels' planes: one load each, 4 bytes (V = float) or 16 (float4). A chunk that lies in one run walks its
// planes, the last one of the layer too; the address arithmetic of a run look-up per load costs more than the load (58 -> 114 3x3 48x8
// x15, whose last chunk has 10 channels: 8.0 -> 6.4 us, quantized inside).
template <typename V>
__device__ __forceinline__ void load16(V (&v)[16], const QuantSource& Q, int c0, int cin, int img, int hw, int p) {
    if (c0 >= Q.first[1] || min(c0 + 16, cin) <= Q.first[1]) {
        const float* ptr = Q.plane(c0, img, hw) + p;
#pragma unroll
        for (int j = 0; j < 16; ++j, ptr += hw) v[j] = c0 + j < cin ? __ldg(reinterpret_cast<const V*>(ptr)) : V{};
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = c0 + j < cin ? __ldg(reinterpret_cast<const V*>(Q.plane(c0 + j, img, hw) + p)) : V{};
    }
}
__device__ __forceinline__ void quantize16(uint32_t addr, const float (&v)[16], const QuantSource& Q) {
    uint32_t w[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) w[g] = quantize4_pack(v[4 * g], v[4 * g + 1], v[4 * g + 2], v[4 * g + 3], Q.scale, Q.half);
    store_chunk(addr, w[0], w[1], w[2], w[3]);
}

// kRowsQuantBuild: the fp32 planes as a tensor [image][channel][pixel]
struct BoxSource {
    CUtensorMap x;
    float scale;
    uint32_t half;
};
template <int BUILD>
using InputOf = std::conditional_t<BUILD == kRowsQuantBuild, BoxSource, std::conditional_t<build_quantizes(BUILD), QuantSource, KernelMaps>>;

// Four pixels of 16 channels -> chunk `chunk` of rows row .. row + 3 of an operand tile.
__device__ __forceinline__ void quantize_quad(const float4 (&v)[16], uint32_t tile, int bkc, int row, int chunk, const QuantSource& Q) {
    uint32_t w[4][4];  // [group of four channels][pixel]
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        uint32_t cw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 f = v[4 * g + j];
            cw[j] = quantize4_pack(f.x, f.y, f.z, f.w, Q.scale, Q.half);
        }
        transpose4x4(cw[0], cw[1], cw[2], cw[3], w[g]);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) store_chunk(operand_chunk(tile, bkc, row + j, chunk), w[0][j], w[1][j], w[2][j], w[3][j]);
}

// Stride-2 halo (UmmaPlan::halo == 2): the input columns under a pixel tile as two planes, one per parity, every row of each. The 8
// pixels of a tile row are then 8 neighbours of the plane that a tap reads, and tile rows are two plane rows apart.
struct ParityHalo {
    int cols[2], rows;
    __host__ __device__ __forceinline__ ParityHalo(int kh, int kw) : cols{kHaloTw + (kw - 1) / 2, kHaloTw + (kw - 2) / 2}, rows(2 * (kHaloTh - 1) + kh) {}
    __host__ __device__ __forceinline__ uint32_t plane_bytes(int i, int bkc) const { return (uint32_t)(rows * cols[i] * bkc); }
    __host__ __device__ __forceinline__ uint32_t second(int bkc) const { return (plane_bytes(0, bkc) + 1023u) & ~1023u; }  // offset of plane 1
    __host__ __device__ __forceinline__ uint32_t stage_bytes(int bkc) const { return second(bkc) + ((plane_bytes(1, bkc) + 1023u) & ~1023u); }
};

// columns of an accumulator an epilogue warp takes at a time
__host__ __device__ __forceinline__ int epi_chunk(const UmmaPlan& p) { return p.bn <= 32 || p.compact ? 16 : 32; }

struct SmemLayout {
    uint32_t b_panel, a_stages, out_slots, floats, bars, tmem_slot, abort_flag, params, total;
};

// ROWS: where finished accumulators of 128 and of 64 channels go.
struct RowsOut {
    CUtensorMap full, half;
};
__host__ __device__ __forceinline__ uint32_t out_slot_bytes(const UmmaPlan& p) { return (uint32_t)p.rows * (p.bn <= 64 ? 64u : 128u); }

__host__ __device__ inline SmemLayout smem_layout(const UmmaPlan& p) {
    SmemLayout L;
    L.b_panel = 0;
    L.a_stages = (uint32_t)p.nkb * p.bn * p.bkc;
    L.out_slots = L.a_stages + (uint32_t)p.stages * (uint32_t)p.a_stage_bytes;
    L.floats = L.out_slots + (p.rows ? (uint32_t)p.out_slots * out_slot_bytes(p) : 0u);
    L.bars = L.floats + (uint32_t)p.boxes * kBoxBytes;
    // barriers: full[stages], empty[stages], b_full, tmem_full[kMaxAccBufs], tmem_empty[kMaxAccBufs], out_full[kOutSlots], out_free[kOutSlots], box_full[boxes], box_free[boxes]
    L.tmem_slot = L.bars + 8u * (2u * p.stages + 1u + 2u * kMaxAccBufs + (p.rows ? 2u * kOutSlots + 2u * p.boxes : 0u));
    L.abort_flag = L.tmem_slot + 8;
    L.params = (L.abort_flag + 8 + 15u) & ~15u;  // scale_in[bn], bias[bn], scale_out[bn]; read as float4
    L.total = L.params + 3u * 4u * p.bn;
    return L;
}

// BUILD 1: compiled for two resident CTAs per SM (at most 102 registers per thread), which small layers need to hide latency;
// BUILD 2: 576 threads (sixteen epilogue warps) for wide tiles with one CTA per SM; BUILD 0: 320 threads, one CTA per SM;
// the one-CTA-per-SM plans of large layers use the build without that register limit.
//
// A launch whose CTAs have one tile each is a serial chain (previous kernel -> activations -> MMAs -> epilogue -> end), so what
// does not need the data stays off it: the producer has its first coordinates, its barrier's byte count and its descriptors
// ready before it waits for the previous kernel and then issues the copy at once (stage and tap counters walk; the divisions
// they replaced took 700 of the 1000 cycles between that wait and the first copy), the MMA issuer and the teardown wait for no
// kernel at all, the epilogue warps work out their pixel before they wait for the accumulator, and tensor memory is freed
// while the last rows are still being requantized.
//
// BUILDs 4 and 5: see kAnyOut.
//
// BUILDs 6, 7 and 8: the operands change places, D[channels, pixels] = W x A^T. Written with pixels as rows, a thread's accumulators belong
// to 16 or 32 channels, whose three parameters each it has to fetch from shared memory for every pixel, and its results are 32 bytes
// of a row of their own, of which a warp's store touches 32: TMEM -> int8 reached 18.9 values per ns and SM that way (ReLU; without
// the stores 31). With channels as rows a thread has the same two channels of every 16 (tcgen05.ld.16x256b) and keeps their parameters in
// registers; stmatrix turns four pixels' bytes into rows of 16 channels in shared memory, and a warp of its own sends a finished tile of
// 128 pixels x 128 channels off as one TMA store: 32.5 values per ns and SM (24 against 18.3 with the general rounding).
// BUILD 8 takes fp32 planes: TMA brings boxes of 16 channels x 64 pixels, ten warps quantize one box each at a time into the tile's operand
// (so that every channel of the layer is computed from one quantized tile, four accumulators of 64 columns at most), and the shared
// memory that up to 128 KB of weights leave is spent on boxes under way: six of them 50.8 us for 256 -> 512 28x28 x128, ten 38.7; by loads into
// registers, which share what is left of L1, 43.3.
//
// BUILD 3: fp32 NCHW input, quantized inside the kernel: warps 10..17 take the TMA producer's place, load the planes, quantize and
// write the operand tiles (with TMA's swizzle) themselves. No int8 copy of the input crosses HBM and no second kernel runs.
template <int OUT, int ACT_BUILD, int BUILD>
__global__ void __launch_bounds__(build_threads(BUILD), BUILD == 1 || BUILD == kCompactBuild || BUILD == kRowsBuild ? 2 : 1)
dense_umma_kernel(const __grid_constant__ InputOf<BUILD> maps, const __grid_constant__ CUtensorMap tmB, const UmmaPlan P,
                  const ConvShape s, const EpilogueParams ep, void* __restrict__ out, uint32_t* __restrict__ status,
                  const __grid_constant__ std::conditional_t<build_rows(BUILD), RowsOut, UmmaMixedOut> mixed) {
    constexpr int ACT = ACT_BUILD & ~kOneScale;
    constexpr bool ONE_SCALE = (ACT_BUILD & kOneScale) != 0, COMPACT = BUILD == kCompactBuild || BUILD == kCompactQuantBuild, QUANT = build_quantizes(BUILD),
                   ROWS = build_rows(BUILD);
    // Pixels of a tile that are loaded and written: 128, or in a compact launch of a 1x1 layer fewer (the MMA's other rows read what
    // the stage happens to hold and nobody reads their sums).
    const int tile_rows = COMPACT ? P.tile_rows : ROWS ? rows_pixels(BUILD) : kTileM;
    const auto writes = [&](int kind) { return OUT == kAnyOut ? P.out_kind == kind : OUT == kind; };
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
    const SmemLayout L = smem_layout(P);
    const uint32_t sB = base + L.b_panel, sA = base + L.a_stages;
    const uint32_t bar_full = base + L.bars, bar_empty = bar_full + 8u * P.stages, bar_b = bar_empty + 8u * P.stages;
    const uint32_t bar_tfull = bar_b + 8, bar_tempty = bar_tfull + 8u * kMaxAccBufs;
    const uint32_t bar_ofull = bar_tempty + 8u * kMaxAccBufs, bar_ofree = bar_ofull + 8u * kOutSlots, bar_xfull = bar_ofree + 8u * kOutSlots,
                   bar_xfree = bar_xfull + 8u * P.boxes;  // (ROWS)
    const int boxes_per_tile = (s.cin + kBoxChannels - 1) / kBoxChannels;  // (ROWS, QUANT)
    const uint32_t acc_mask = (uint32_t)P.acc_bufs - 1u, acc_shift = P.acc_bufs == 8 ? 3u : P.acc_bufs == 4 ? 2u : 1u;  // 2, 4 or 8 accumulators in TMEM
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(base_ptr + L.tmem_slot);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(base_ptr + L.abort_flag);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_tile = blockIdx.x % P.n_tiles;
    const int m_first = blockIdx.x / P.n_tiles, m_step = gridDim.x / P.n_tiles;
    // ROWS: accumulators of a pixel tile, 128 channels each, the last one of the layer 64 where that holds what is left
    const int cols_left = s.cout_pad - n_tile * P.bn, my_cols = cols_left < P.bn ? cols_left : P.bn;
    const int blocks = ROWS && BUILD != kRowsBuild ? (my_cols + kTileM - 1) / kTileM : 1;
    const uint32_t a_stage_bytes = (uint32_t)P.a_stage_bytes, b_tile_bytes = (uint32_t)P.bn * P.bkc;
    // halo mode: the 8 pixels of one tile row are one 8-row operand group; groups (tile rows) are one halo row apart
    const int halo_w = kHaloTw + s.kw - 1, halo_h = kHaloTh + s.kh - 1;
    const ParityHalo parity(s.kh, s.kw);
    // pipeline stages one pixel tile consumes (a gathered layer's stage holds all the K blocks of a tile: one barrier round
    // trip per tile instead of one per 32-channel block)
    const int loads_per_tile = ROWS && QUANT ? 1 : P.halo ? P.ncb : (P.gather && P.gather_whole ? 1 : P.nkb);

    // Tensor memory first, and only then may the next kernel start: a CTA of it that shared this SM and allocated before this one
    // would hold the columns this one waits for while it waits for this kernel to end.
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)),
                     "r"((uint32_t)P.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        if (!ROWS || !P.late) pdl_launch_dependents();
    }
    if (threadIdx.x == 0) {
        prefetch_tensormap(&tmB);
        if constexpr (!QUANT)
#pragma unroll 1
            for (int i = 0; i < (P.gather > 0 ? P.gather : 1); ++i) prefetch_tensormap(&maps.tm[i]);
#pragma unroll 1
        for (int i = 0; i < P.stages; ++i) {
            mbar_init(bar_full + 8u * i, ROWS && QUANT ? kBoxWarps : QUANT ? kQuantWarps : 1);
            mbar_init(bar_empty + 8u * i, 1);
        }
        mbar_init(bar_b, 1);
#pragma unroll 1
        for (int i = 0; i < P.acc_bufs; ++i) {
            mbar_init(bar_tfull + 8u * i, 1);
            mbar_init(bar_tempty + 8u * i, ROWS ? (uint32_t)team_warps(BUILD)
                                                : (uint32_t)(tile_rows + 31) / 32u * (uint32_t)((P.bn + epi_chunk(P) - 1) / epi_chunk(P)));  // one arrival per lane quarter and column chunk
        }
        if constexpr (ROWS) {
            prefetch_tensormap(my_cols > 64 ? &mixed.full : &mixed.half);
#pragma unroll 1
            for (int i = 0; i < P.out_slots; ++i) {
                mbar_init(bar_ofull + 8u * i, (uint32_t)team_warps(BUILD));
                mbar_init(bar_ofree + 8u * i, 1);
            }
#pragma unroll 1
            for (int i = 0; i < P.boxes; ++i) {
                mbar_init(bar_xfull + 8u * i, 1);
                mbar_init(bar_xfree + 8u * i, 1);
            }
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the weight panel does not depend on the previous kernel: start loading it before waiting for that kernel
        mbar_expect_tx(bar_b, (uint32_t)P.nkb * b_tile_bytes);
#pragma unroll 1
        for (int kb = 0; kb < P.nkb; ++kb)
            if constexpr (ROWS && QUANT) {  // (a panel of up to 512 channels: 64 at a time)
#pragma unroll 1
                for (int c = 0; c < P.bn; c += 64) tma_load_2d(&tmB, bar_b, sB + kb * b_tile_bytes + (uint32_t)(c * P.bkc), kb * P.bkc, n_tile * P.bn + c);
            } else {
                tma_load_2d(&tmB, bar_b, sB + kb * b_tile_bytes, kb * P.bkc, n_tile * P.bn);
            }
    }
    {
        float* sp = reinterpret_cast<float*>(base_ptr + L.params);
#pragma unroll 1
        for (int i = threadIdx.x; i < P.bn; i += (int)blockDim.x) {
            const int c = n_tile * P.bn + i;
            const bool in = c < s.cout_pad;
            sp[i] = in ? ep.scale_in[c] : 0.f;
            sp[P.bn + i] = in ? bias_or_neutral(ep, c) : 0.f;
            sp[2 * P.bn + i] = in ? ep.scale_out[c] : 0.f;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if constexpr (ROWS && QUANT) {
            if (elect_one()) {
                // ---- TMA producer (fp32 planes): box b of the CTA goes to quantizing warp b % kBoxWarps, whose boxes have places of their own ----
                pdl_wait();
                uint32_t at = 0, phase = 1;
                bool ok = true;
                for (int m = m_first; ok && m < P.m_tiles; m += m_step) {
                    const int img = (int)fast_div((uint32_t)m, P.div_img), p0 = (m - img * P.tiles_x) * rows_pixels(BUILD);
                    for (int c = 0; c < s.cin; c += kBoxChannels) {
                        if (!mbar_wait(bar_xfree + 8u * at, phase, abort_flag, status, 256u, P.wait_ns)) { ok = false; break; }
                        mbar_expect_tx(bar_xfull + 8u * at, kBoxBytes);
                        tma_load_3d(&maps.x, bar_xfull + 8u * at, base + L.floats + at * kBoxBytes, p0, c, img);
                        if (++at == (uint32_t)P.boxes) { at = 0; phase ^= 1u; }
                    }
                }
                if (!ok) {
                    const unsigned long long t0 = globaltimer_ns();  // (as below)
                    while (globaltimer_ns() - t0 < 1000000ull) {}
                }
            }
        }
        if constexpr (!QUANT)
        if (elect_one()) {
            // ---- TMA producer (activations; the weights were requested during set-up) ----
            uint32_t st = 0, phase = 1;  // stage, and the parity that says it is free (the first round finds every stage free)
            bool ok = true, waited = false;
            const uint32_t load_bytes = P.gather && P.gather_whole ? (uint32_t)(tile_rows * P.bkc * P.nkb)
                                        : P.halo == 2               ? parity.plane_bytes(0, P.bkc) + parity.plane_bytes(1, P.bkc)
                                        : P.halo                    ? (uint32_t)(halo_w * halo_h * P.bkc)
                                                                    : (uint32_t)(tile_rows * P.bkc);
            for (int m = m_first; ok && m < P.m_tiles; m += m_step) {
                int img = 0, y0 = 0, x0 = m * tile_rows;
                if (!P.flat) {
                    img = (int)fast_div((uint32_t)m, P.div_img);
                    const int r = m - img * P.tiles_x * P.tiles_y, ty = (int)fast_div((uint32_t)r, P.div_tx);
                    y0 = ty * P.th * s.sh - s.ph;
                    x0 = (r - ty * P.tiles_x) * P.tw * s.sw - s.pw;
                }
                int cb = 0, kx = 0, ky = 0;  // per-tap loads: channel block and tap of the next box
                for (int kb = 0; kb < loads_per_tile; ++kb) {
                    const uint32_t full = bar_full + 8u * st, dst = sA + st * a_stage_bytes;
                    if (!mbar_wait(bar_empty + 8u * st, phase, abort_flag, status, 1u, P.wait_ns)) { ok = false; break; }
                    mbar_expect_tx(full, load_bytes);
                    if (!waited) {
                        pdl_wait();  // from here on the kernel reads what the previous one wrote
                        waited = true;
                    }
                    if (P.gather && P.gather_whole) {
#pragma unroll 1
                        for (int g = 0; g < P.nkb; ++g)
                            tma_load_4d(&maps.tm[maps.block_src[g]], full, dst + (uint32_t)(g * kTileM * P.bkc), (int)maps.block_x[g], x0, 0, 0);
                    } else if (P.gather) {
                        // K block kb = 32 channels of one of the source tensors (channels past that tensor's end arrive as zeros)
                        tma_load_4d(&maps.tm[maps.block_src[kb]], full, dst, (int)maps.block_x[kb], x0, 0, 0);
                    } else if (!COMPACT && !ROWS && P.halo == 2) {
                        tma_load_4d(&maps.tm[0], full, dst, kb * P.bkc, x0, y0, img);
                        tma_load_4d(&maps.tm[1], full, dst + parity.second(P.bkc), kb * P.bkc, x0 + 1, y0, img);
                    } else if (!ROWS && P.halo) {
                        // the (8 + kw - 1) x (16 + kh - 1) pixels under the tile, one channel block; out-of-image pixels arrive as zeros
                        tma_load_4d(&maps.tm[0], full, dst, kb * P.bkc, x0, y0, img);
                    } else {
                        tma_load_4d(&maps.tm[0], full, dst, cb * P.bkc, x0 + kx * s.dw, y0 + ky * s.dh, img);
                        if (++cb == P.ncb) {
                            cb = 0;
                            if (++kx == s.kw) { kx = 0; ++ky; }
                        }
                    }
                    if (++st == (uint32_t)P.stages) { st = 0; phase ^= 1u; }
                }
            }
            if (!ok) {
                // let bulk copies already in flight land before the CTA's shared memory is released
                const unsigned long long t0 = globaltimer_ns();
                while (globaltimer_ns() - t0 < 1000000ull) {}
            }
        }
    } else if (warp == 1) {
        // (BUILD 3: the uniform registers' copies of an elected issuer's offsets would take the quantizers' registers, 36 bytes spilled: 60
        // -> 167 48x14 x348 35.1 us, this way 31.2; of 170 layers on fp32 input none is slower than with an elected one)
        if (BUILD == kQuantBuild ? lane == 0 : elect_one()) {
            // ---- MMA issuer ----
            bool ok = mbar_wait(bar_b, 0, abort_flag, status, 16u, P.wait_ns);
            tc_fence_after();
            pdl_wait();  // (no wait below is counted against its limit while the previous kernel still runs)
            uint32_t st = 0, phase = 0, tile_i = 0;  // (tile_i counts accumulators: ROWS has several per tile)
            const uint32_t idesc_half = P.idesc - ((uint32_t)(kTileM >> 5) << 24);  // ROWS, 64 rows
            for (int m = m_first; ok && m < P.m_tiles; m += m_step, tile_i += (uint32_t)blocks) {
                const uint32_t buf = tile_i & acc_mask, use = tile_i >> acc_shift;
                if (!mbar_wait(bar_tempty + 8u * buf, (use & 1u) ^ 1u, abort_flag, status, 4u, P.wait_ns)) { ok = false; break; }
                const uint32_t d = tmem_base + buf * (uint32_t)P.acc_stride;
                // ROWS: the tile's other accumulators
                constexpr int kMore = BUILD == kRowsQuantBuild ? kRowsMaxBlocks - 1 : BUILD == kRowsWideBuild ? 1 : 0;
                uint32_t more[kMore + 1];
#pragma unroll
                for (int b = 0; b < kMore; ++b) {
                    if (b + 1 >= blocks) break;
                    const uint32_t unit = tile_i + 1u + (uint32_t)b, bb = unit & acc_mask;
                    if (ok && !mbar_wait(bar_tempty + 8u * bb, ((unit >> acc_shift) & 1u) ^ 1u, abort_flag, status, 4u, P.wait_ns)) ok = false;
                    more[b] = tmem_base + bb * (uint32_t)P.acc_stride;
                }
                if (!ok) break;
                tc_fence_after();
                // pixels: the operand with the tile's pixels as rows; weights: the one with channels as rows
                auto mma = [&](uint64_t pixels, uint64_t weights, uint32_t accumulate) {
                    if constexpr (ROWS) {
                        umma_i8(d, weights, pixels, blocks > 1 || my_cols > 64 ? P.idesc : idesc_half, accumulate);
#pragma unroll
                        for (int b = 0; b < kMore; ++b)
                            if (b + 1 < blocks)
                                umma_i8(more[b], weights + (uint32_t)(b + 1) * ((uint32_t)(kTileM * P.bkc) >> 4), pixels,
                                        my_cols > (b + 1) * kTileM + 64 ? P.idesc : idesc_half, accumulate);
                    } else {
                        umma_i8(d, pixels, weights, P.idesc, accumulate);
                    }
                };
                for (int kb = 0; kb < loads_per_tile; ++kb) {
                    if (!mbar_wait(bar_full + 8u * st, phase, abort_flag, status, 2u, P.wait_ns)) { ok = false; break; }
                    tc_fence_after();
                    if (!COMPACT && !QUANT && !ROWS && P.halo == 2) {
                        // a tap of column kx reads plane kx & 1, from column kx >> 1 on
                        const uint32_t tile = sA + st * a_stage_bytes, px_step = (uint32_t)P.bkc >> 4;
                        const uint64_t a0 = make_smem_desc(tile, P.bkc, 2 * parity.cols[0] * P.bkc);
                        const uint64_t a1 = make_smem_desc(tile + parity.second(P.bkc), P.bkc, 2 * parity.cols[1] * P.bkc);
                        const uint64_t b0 = make_smem_desc(sB + kb * b_tile_bytes, P.bkc);
                        const uint32_t b_tap_step = ((uint32_t)P.ncb * b_tile_bytes) >> 4;
                        auto tap = [&](int ky, int kx, int J, uint32_t b_off) {
                            const uint32_t a_off = (uint32_t)(ky * parity.cols[kx & 1] + (kx >> 1)) * px_step;
                            const uint64_t a = ((kx & 1) ? a1 : a0) + a_off;
#pragma unroll
                            for (int j = 0; j < 4; ++j)
                                if (j < J) mma(a + 2u * j, b0 + b_off + 2u * j, (kb | ky | kx | j) != 0 ? 1u : 0u);
                        };
                        const int J = P.bkc / 32;
                        if (s.kh == 3 && s.kw == 3) {
                            uint32_t b_off = 0;
#pragma unroll 1
                            for (int ky = 0; ky < 3; ++ky)  // (a loop for the same reason)
#pragma unroll
                                for (int kx = 0; kx < 3; ++kx, b_off += b_tap_step) tap(ky, kx, J, b_off);
                        } else {
#pragma unroll 1
                            for (int i = 0, ky = 0, kx = 0; i < P.taps; ++i) {
                                tap(ky, kx, J, (uint32_t)i * b_tap_step);
                                if (++kx == s.kw) { kx = 0; ++ky; }
                            }
                        }
                    } else if (!ROWS && P.halo) {
                        // every filter tap reads the same halo tile through a view shifted by (ky, kx) pixels
                        // (one thread issues all of these back to back, so the per-tap descriptors are the base descriptors plus
                        // an offset in their 16-byte address field, not rebuilt from scratch)
                        const uint64_t a0 = make_smem_desc(sA + st * a_stage_bytes, P.bkc, halo_w * P.bkc);
                        const uint64_t b0 = make_smem_desc(sB + kb * b_tile_bytes, P.bkc);
                        const uint32_t b_tap_step = ((uint32_t)P.ncb * b_tile_bytes) >> 4, a_px_step = (uint32_t)P.bkc >> 4;
                        uint32_t accumulate = kb != 0 ? 1u : 0u, a_row = 0, b_off = 0;
                        if ((!COMPACT || QUANT) && s.kh == 3 && s.kw == 3) {
                            // the common filter: loops unrolled, every descriptor the base's low word plus a constant (the address
                            // field cannot carry), so that the one issuing thread spends its time issuing. The rows of 128-channel
                            // blocks stay a loop: with all 36 MMAs in line the descriptors' offsets are worked out ahead of the tile
                            // loop and take the registers of the 96-register builds' epilogue (up to 44 bytes spilled; 64 -> 64 56x56
                            // x256 int8, ReLU: 42.7 us, this way 38.1; 32 -> 64 80x80 x128 35.5 / 30.9)
                            const uint32_t a_lo = (uint32_t)a0, b_lo = (uint32_t)b0;
                            const uint64_t a_hi = a0 & 0xFFFFFFFF00000000ull, b_hi = b0 & 0xFFFFFFFF00000000ull;
                            auto taps = [&](auto steps) {
                                constexpr int J = decltype(steps)::value;
                                uint32_t al = a_lo, bl = b_lo;
#pragma unroll (J == 4 ? 1 : 3)
                                for (int ky = 0; ky < 3; ++ky, al += 2u * J * (kHaloTw + 2))
#pragma unroll
                                    for (int kx = 0; kx < 3; ++kx, bl += b_tap_step)
#pragma unroll
                                        for (int j = 0; j < J; ++j) {
                                            mma(a_hi | (uint64_t)(al + 2u * (J * kx + j)), b_hi | (uint64_t)(bl + 2u * j), accumulate);
                                            accumulate = 1u;
                                        }
                            };
                            if (P.bkc == 128) taps(std::integral_constant<int, 4>{});
                            else if (P.bkc == 64) taps(std::integral_constant<int, 2>{});
                            else taps(std::integral_constant<int, 1>{});
                        } else
                        for (int ky = 0; ky < s.kh; ++ky, a_row += (uint32_t)halo_w * a_px_step) {
                            uint32_t a_off = a_row;
                            for (int kx = 0; kx < s.kw; ++kx, a_off += a_px_step, b_off += b_tap_step) {
#pragma unroll (COMPACT ? 1 : 4)
                                for (int j = 0; j < P.bkc / 32; ++j) {
                                    mma(a0 + a_off + 2u * j, b0 + b_off + 2u * j, accumulate);
                                    accumulate = 1u;
                                }
                            }
                        }
                    } else if constexpr (ROWS && QUANT) {
                        // one stage holds all the K blocks of the tile, 64 pixels each
                        const uint64_t a0 = make_smem_desc(sA + st * a_stage_bytes, P.bkc), b0 = make_smem_desc(sB, P.bkc);
                        const uint32_t a_step = (uint32_t)(rows_pixels(BUILD) * P.bkc) >> 4, b_step = b_tile_bytes >> 4;
#pragma unroll 1
                        for (int g = 0; g < P.nkb; ++g)
#pragma unroll 1
                            for (int j = 0; j < P.bkc / 32; ++j)
                                mma(a0 + (uint32_t)g * a_step + 2u * j, b0 + (uint32_t)g * b_step + 2u * j, (g | j) != 0 ? 1u : 0u);
                    } else if (P.gather && P.gather_whole) {
                        // one stage holds all the K blocks of the tile; per block only the low words of the two descriptors move
                        const uint64_t a0 = make_smem_desc(sA + st * a_stage_bytes, P.bkc), b0 = make_smem_desc(sB, P.bkc);
                        const uint32_t a_lo = (uint32_t)a0, b_lo = (uint32_t)b0;
                        const uint64_t a_hi = a0 & 0xFFFFFFFF00000000ull, b_hi = b0 & 0xFFFFFFFF00000000ull;
                        const uint32_t a_step = (uint32_t)(kTileM * P.bkc) >> 4, b_step = b_tile_bytes >> 4;
                        uint32_t ao = 0, bo = 0;
#pragma unroll 1
                        for (int g = 0; g < P.nkb; ++g, ao += a_step, bo += b_step)
#pragma unroll 1
                            for (int j = 0; j < P.bkc / 32; ++j)
                                mma(a_hi | (uint64_t)(a_lo + ao + 2u * j), b_hi | (uint64_t)(b_lo + bo + 2u * j), (g | j) != 0 ? 1u : 0u);
                    } else {
                        const uint64_t adesc = make_smem_desc(sA + st * a_stage_bytes, P.bkc);
                        const uint64_t bdesc = make_smem_desc(sB + kb * b_tile_bytes, P.bkc);
                        const uint32_t a_lo = (uint32_t)adesc, b_lo = (uint32_t)bdesc;
                        const uint64_t a_hi = adesc & 0xFFFFFFFF00000000ull, b_hi = bdesc & 0xFFFFFFFF00000000ull;
                        auto steps = [&](auto n) {
                            constexpr int J = decltype(n)::value;
#pragma unroll
                            for (int j = 0; j < J; ++j) mma(a_hi | (uint64_t)(a_lo + 2u * j), b_hi | (uint64_t)(b_lo + 2u * j), (kb | j) != 0 ? 1u : 0u);
                        };
                        if (COMPACT) {
#pragma unroll 1
                            for (int j = 0; j < P.bkc / 32; ++j) mma(a_hi | (uint64_t)(a_lo + 2u * j), b_hi | (uint64_t)(b_lo + 2u * j), (kb | j) != 0 ? 1u : 0u);
                        } else if (P.bkc == 128) steps(std::integral_constant<int, 4>{});
                        else if (P.bkc == 64) steps(std::integral_constant<int, 2>{});
                        else steps(std::integral_constant<int, 1>{});
                    }
                    umma_commit(bar_empty + 8u * st);  // frees the A stage once these MMAs have read it
                    if (++st == (uint32_t)P.stages) { st = 0; phase ^= 1u; }
                }
                if (!ok) break;
                umma_commit(bar_tfull + 8u * buf);  // accumulator complete
                if (ROWS && !QUANT && blocks > 1) umma_commit(bar_tfull + 8u * ((tile_i + 1) & acc_mask));
                if constexpr (ROWS && QUANT)
#pragma unroll 1
                    for (int b = 1; b < blocks; ++b) umma_commit(bar_tfull + 8u * ((tile_i + (uint32_t)b) & acc_mask));
            }
            // every accumulator read for the last time: the tensor memory can go back
            for (uint32_t b = 0; ok && b <= acc_mask && b < tile_i; ++b)
                ok = mbar_wait(bar_tempty + 8u * b, (((tile_i - 1 - b) >> acc_shift) & 1u), abort_flag, status, 4u, P.wait_ns);
            if (!ok) *abort_flag = 1;
        }
        __syncwarp();
        // an aborted CTA frees the tensor memory only when all other warps have left (exited threads count as arrived)
        if (*abort_flag) __syncthreads();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)P.tmem_cols) : "memory");
    } else if (ROWS && QUANT && warp > 2 + kMaxEpiWarps) {
        if constexpr (ROWS && QUANT) {
            // ---- quantizers: four pixels of eight channels per thread. Every warp waits for every tile's stage and arrives on its barrier
            // once, after its last box of the tile or without one (fewer than kBoxWarps boxes): the tile is multiplied, and its stage
            // freed again, only when all of them have seen the stage free, so that none misses a phase of bar_empty ----
            const int qw = warp - (3 + kMaxEpiWarps), quad = lane & 15, upper = lane >> 4, per_block = 31 - __clz(P.bkc >> 4);
            const uint32_t words_at = base + L.floats + (uint32_t)(upper * 8 * rows_pixels(BUILD) * 4 + quad * 16);
            uint32_t st = 0, phase = 1, at = (uint32_t)qw, xphase = 0;
            int c = qw;  // this warp's next box, counted from the tile's first
            bool ok = true;
            pdl_wait();  // (as the issuer: the previous kernel's time does not count against the limits of the waits below)
            for (int m = m_first; ok && m < P.m_tiles; m += m_step) {
                bool waited = false;
                for (; c < boxes_per_tile; c += kBoxWarps) {
                    float4 v[8];
                    if (!mbar_wait_warp(bar_xfull + 8u * at, xphase, abort_flag, status, 512u, P.wait_ns)) { ok = false; break; }
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[j].x), "=f"(v[j].y), "=f"(v[j].z), "=f"(v[j].w)
                                     : "r"(words_at + at * kBoxBytes + (uint32_t)(j * rows_pixels(BUILD) * 4)) : "memory");
                    if (!waited && !mbar_wait_warp(bar_empty + 8u * st, phase, abort_flag, status, 1u, P.wait_ns)) { ok = false; break; }
                    waited = true;
                    uint32_t w[2][4];  // [group of four channels][pixel]
#pragma unroll
                    for (int g = 0; g < 2; ++g) {
                        uint32_t cw[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) cw[j] = quantize4_pack(v[4 * g + j].x, v[4 * g + j].y, v[4 * g + j].z, v[4 * g + j].w, maps.scale, maps.half);
                        transpose4x4(cw[0], cw[1], cw[2], cw[3], w[g]);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_xfree + 8u * at);  // the box is read
                    at += kBoxWarps;
                    if (at >= (uint32_t)P.boxes) { at = (uint32_t)qw; xphase ^= 1u; }
                    const uint32_t block = sA + st * a_stage_bytes + (uint32_t)((c >> per_block) * rows_pixels(BUILD) * P.bkc);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(operand_chunk(block, P.bkc, quad * 4 + j, c & ((1 << per_block) - 1)) + (uint32_t)(upper * 8)),
                                     "r"(w[0][j]), "r"(w[1][j]) : "memory");
                }
                if (ok && !waited && !mbar_wait_warp(bar_empty + 8u * st, phase, abort_flag, status, 1u, P.wait_ns)) ok = false;
                if (!ok) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tile's writes -> the MMA's reads
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8u * st);
                c -= boxes_per_tile;
                if (++st == (uint32_t)P.stages) { st = 0; phase ^= 1u; }
            }
        }
    } else if (QUANT && !ROWS && warp >= 2 + kMaxEpiWarps) {
        if constexpr (QUANT && !ROWS) {
            // ---- quantizers: warp q takes every eighth (16 channels, 32 pixels or pixel quads) item of a stage ----
            const int qw = warp - (2 + kMaxEpiWarps), chunks = P.bkc >> 4, hw = s.h * s.w;
            const long total_pix = (long)s.n * hw;
            uint32_t st = 0, phase = 1;
            int turn = qw;  // a stage of fewer than eight items starts with another warp each time
            bool ok = true;
            pdl_wait();
            for (int m = m_first; ok && m < P.m_tiles; m += m_step) {
                int img = 0, y0 = 0, x0 = 0;
                if (!P.flat) {
                    img = (int)fast_div((uint32_t)m, P.div_img);
                    const int r = m - img * P.tiles_x * P.tiles_y, ty = (int)fast_div((uint32_t)r, P.div_tx);
                    y0 = ty * P.th - s.ph;
                    x0 = (r - ty * P.tiles_x) * P.tw - s.pw;
                }
                for (int kb = 0; kb < loads_per_tile; ++kb) {
                    if (!mbar_wait(bar_empty + 8u * st, phase, abort_flag, status, 1u, P.wait_ns)) { ok = false; break; }
                    const uint32_t tile = sA + st * a_stage_bytes;
                    if (P.flat && maps.vec) {
                        const int ch = turn & 7, c0 = kb * P.bkc + ch * 16;
                        const long gp = (long)m * tile_rows + lane * 4;  // four pixels of one image
                        if (ch < chunks && c0 < s.cin && gp < total_pix && lane * 4 < tile_rows) {
                            const int im = (int)fast_div((uint32_t)gp, P.div_plane), p = (int)(gp - (long)im * hw);
                            float4 v[16];
                            load16(v, maps, c0, s.cin, im, hw, p);
                            quantize_quad(v, tile, P.bkc, lane * 4, ch, maps);
                        }
                    } else {
                        // pixel by pixel: flat tiles of any alignment, and halo tiles (out-of-image pixels are zeros)
                        const int pixels = P.flat ? tile_rows : halo_w * halo_h, items = ((pixels + 31) >> 5) * chunks, shift = 31 - __clz(chunks);
                        for (int it = turn & 7; it < items; it += 2 * kQuantWarps) {
                            float v[2][16];
                            uint32_t dst[2];
                            bool have[2];
#pragma unroll
                            for (int u = 0; u < 2; ++u) {
                                const int item = it + u * kQuantWarps, ch = item & (chunks - 1), row = (item >> shift) * 32 + lane, c0 = kb * P.bkc + ch * 16;
                                have[u] = item < items && row < pixels && c0 < s.cin;
                                dst[u] = operand_chunk(tile, P.bkc, row, ch);
                                int im = img, p;
                                bool in;
                                if (P.flat) {
                                    const long gp = (long)m * tile_rows + row;
                                    in = gp < total_pix;
                                    im = (int)fast_div((uint32_t)gp, P.div_plane);
                                    p = (int)(gp - (long)im * hw);
                                } else {
                                    const int hy = (int)fast_div((uint32_t)row, maps.div_halo), iy = y0 + hy, ix = x0 + row - hy * halo_w;
                                    in = iy >= 0 && iy < s.h && ix >= 0 && ix < s.w;
                                    p = iy * s.w + ix;
                                }
                                if (have[u] && in) {
                                    load16(v[u], maps, c0, s.cin, im, hw, p);
                                } else {
#pragma unroll
                                    for (int j = 0; j < 16; ++j) v[u][j] = 0.f;
                                }
                            }
#pragma unroll
                            for (int u = 0; u < 2; ++u)
                                if (have[u]) quantize16(dst[u], v[u], maps);
                        }
                    }
                    turn += chunks;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // these writes -> the MMA's reads
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_full + 8u * st);
                    if (++st == (uint32_t)P.stages) { st = 0; phase ^= 1u; }
                }
            }
        }
    } else if (ROWS && warp == 2 + P.epi_warps) {
        if constexpr (ROWS) {
            if (elect_one()) {
                // ---- finished tiles: one TMA store each (what lies outside the tensor is clipped) ----
                pdl_wait();  // the outputs may still be read by the previous kernel
                uint32_t unit = 0;
                bool ok = true;
                for (int m = m_first; ok && m < P.m_tiles; m += m_step) {
                    const int img = QUANT ? (int)fast_div((uint32_t)m, P.div_img) : 0, p0 = (m - (QUANT ? img * P.tiles_x : 0)) * rows_pixels(BUILD);
                    for (int blk = 0; blk < blocks; ++blk, ++unit) {
                        const uint32_t slot = unit & ((uint32_t)P.out_slots - 1u), use = unit / (uint32_t)P.out_slots;
                        if (!mbar_wait(bar_ofull + 8u * slot, use & 1u, abort_flag, status, 64u, P.wait_ns)) { ok = false; break; }
                        tma_store_3d(my_cols - blk * kTileM > 64 ? &mixed.full : &mixed.half, base + L.out_slots + slot * out_slot_bytes(P),
                                     n_tile * P.bn + blk * kTileM, p0, img);
                        bulk_commit();
                        // A slot is free when its store has been read, 0.5 us after it was issued. With two slots a team waits for that; with
                        // four the next tile's store is issued first (64 -> 256 56x56 x128: one at a time 35.4 us, two 27.7).
                        if (P.out_slots == kOutSlots) {
                            bulk_wait_read<1>();
                            if (unit > 0) mbar_arrive(bar_ofree + 8u * ((unit - 1u) & (kOutSlots - 1)));
                        } else {
                            bulk_wait_read<0>();
                            mbar_arrive(bar_ofree + 8u * slot);
                        }
                    }
                }
                bulk_wait_all();
            }
        }
    } else if (ROWS) {
        if constexpr (ROWS) {
            // ---- epilogue warps, channels as rows. A team of eight (two per lane quarter; of four where tiles are 64 pixels) takes an
            // accumulator; two teams take them in turn, so that a warp has one block's channels for good (with more than two blocks per
            // tile it changes them), and one team's arithmetic fills the other's waits ----
            constexpr uint32_t teams = BUILD == kRowsBuild ? 1 : 2;
            const int q = warp & 3, sub = team_warps(BUILD) == 8 ? ((warp - 2) >> 2) & 1 : 0;
            const uint32_t team = teams == 2 ? (uint32_t)(warp - 2) / (uint32_t)team_warps(BUILD) : 0u;
            int blk = 0, left, c0;  // accumulator block; channels from its first one on, this quarter's first
            bool hi;                // 16 channels at a time: the quarter's first, and its second
            uint32_t row_bytes, at_lo, at_hi;
            const uint32_t half = half_bits(ep.rounding);
            float2 si[2][2], bi[2][2], so[2][2];  // [first / second 16][channel lane / 4, + 8], each twice: for two pixels
            auto take_block = [&](int b) {
                blk = b;
                left = my_cols - blk * kTileM;
                const int per_q = left > 64 ? 32 : 16;  // rows of a quarter (64-row accumulators: its first 16 lanes)
                c0 = q * per_q;
                hi = per_q == 32 && c0 + 16 < left;
                const float* sp = reinterpret_cast<const float*>(base_ptr + L.params);
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int c = blk * kTileM + c0 + (per_q == 32 ? h * 16 : 0) + j * 8 + (lane >> 2);
                        si[h][j] = make_float2(sp[c], sp[c]);
                        bi[h][j] = make_float2(sp[P.bn + c], sp[P.bn + c]);
                        so[h][j] = make_float2(sp[2 * P.bn + c], sp[2 * P.bn + c]);
                    }
                // one byte per channel and row; the 16-byte chunks of a row trade places by the row's number, as the store's swizzle has it
                row_bytes = 4u * (uint32_t)per_q;
                const uint32_t swz = per_q == 32 ? (uint32_t)lane & 7u : ((uint32_t)lane >> 1) & 3u, chunk = (uint32_t)c0 >> 4;
                const uint32_t row0 = base + L.out_slots + ((uint32_t)(sub * 64) + (uint32_t)lane) * row_bytes;
                at_lo = row0 + ((chunk ^ swz) << 4);
                at_hi = row0 + (((chunk + 1u) ^ swz) << 4);
            };
            take_block(blocks > 1 ? (int)team : 0);
            const uint32_t t_lane = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(sub * 64);
            const uint32_t slot_bytes = out_slot_bytes(P), slot_mask = (uint32_t)P.out_slots - 1u, slot_shift = P.out_slots == 4 ? 2u : 1u;
            auto emit = [&](const int (&a)[16], int h, uint32_t at) {
                uint32_t w[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    float2 y[2];
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float2 t = __ffma2_rn(make_float2(__int2float_rn(a[4 * g + 2 * j]), __int2float_rn(a[4 * g + 2 * j + 1])), si[h][j], bi[h][j]);
                        y[j] = make_float2(activate_t<ACT>(t.x, ep.act_param0), activate_t<ACT>(t.y, ep.act_param0));
                    }
                    if constexpr (ACT == ACT_POS) {
                        w[g] = requant4_pos(y[0], so[h][0], y[1], so[h][1]);
                    } else {
                        const int2 qa = round2(__fmul2_rn(y[0], so[h][0]), half), qb = round2(__fmul2_rn(y[1], so[h][1]), half);
                        w[g] = pack_sat_s8x4(qa.x, qa.y, qb.x, qb.y);
                    }
                }
                stmatrix_t8(at, w);
            };
            pdl_wait();  // (as the issuer)
            const uint32_t units = m_first < P.m_tiles ? (uint32_t)((P.m_tiles - 1 - m_first) / m_step + 1) * (uint32_t)blocks : 0u;
            for (uint32_t unit = team; unit < units; unit += teams) {
                if (QUANT && blocks > 2 && unit != team) take_block(blk + 2 < blocks ? blk + 2 : blk + 2 - blocks);
                const uint32_t buf = unit & acc_mask, use = unit >> acc_shift, slot = unit & slot_mask;
                const uint32_t taddr = t_lane + buf * (uint32_t)P.acc_stride, out_at = slot * slot_bytes;
                // A lane whose wait has run out goes on with the others, over sums that mean nothing, to the warp's last unit (the abort flag is
                // up, so that no further wait lasts, and the call reports it): what follows wants all 32 lanes. Leaving the loop by a vote costs
                // 58 -> 58 40x40 x256 0.45 us, this way, which joins the lanes behind each wait, 0.2 of 10.4.
                (void)mbar_wait(bar_tfull + 8u * buf, use & 1u, abort_flag, status, 8u, P.wait_ns);
                tc_fence_after();
                // 32 pixels x 16 channels at a time, the next ones on their way while these are computed
                int v[2][16];
                if (c0 < left) tmem_ld16x256(taddr, v[0]);
                (void)mbar_wait(bar_ofree + 8u * slot, ((unit >> slot_shift) & 1u) ^ 1u, abort_flag, status, 128u, P.wait_ns);
                tmem_wait_ld16(v[0]);
                if (hi) {
                    tmem_ld16x256(taddr + (16u << 16), v[1]);
                    emit(v[0], 0, at_lo + out_at);
                    tmem_wait_ld16(v[1]);
                    tmem_ld16x256(taddr + 32u, v[0]);
                    emit(v[1], 1, at_hi + out_at);
                    tmem_wait_ld16(v[0]);
                    tmem_ld16x256(taddr + (16u << 16) + 32u, v[1]);
                    emit(v[0], 0, at_lo + out_at + 32u * row_bytes);
                    tmem_wait_ld16(v[1]);
                } else if (c0 < left) {
                    tmem_ld16x256(taddr + 32u, v[1]);
                    emit(v[0], 0, at_lo + out_at);
                    tmem_wait_ld16(v[1]);
                }
                tc_fence_before();  // the accumulator is read
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_tempty + 8u * buf);
                if (hi) emit(v[1], 1, at_hi + out_at + 32u * row_bytes);
                else if (c0 < left) emit(v[1], 0, at_lo + out_at + 32u * row_bytes);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // these writes -> the TMA store's reads
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_ofull + 8u * slot);
            }
        }
    } else if constexpr (!ROWS) {
        // ---- epilogue warps ----
        const int q = warp & 3;            // TMEM lane quarter this warp may read
        const int sub = (warp - 2) >> 2;   // which of the epi_warps/4 warps sharing that quarter
        const int chunk = COMPACT ? 16 : epi_chunk(P), n_chunks = (P.bn + chunk - 1) / chunk, nsub = P.epi_warps / 4;
        const int row = q * 32 + lane;
        const int row_y = row >> (31 - __clz(P.tw)), row_x = row & (P.tw - 1);  // (tw is a power of two)
        const long plane = (long)s.oh * s.ow;
        const long total_pix = (long)s.n * plane;
        const float* s_si = reinterpret_cast<const float*>(base_ptr + L.params);
        const float* s_bi = s_si + P.bn;
        const float* s_so = s_bi + P.bn;
        const int c_base = n_tile * P.bn;  // the output channel of accumulator column 0
        const uint32_t half = half_bits(ep.rounding);
        uint32_t tile_i = 0;
        // The warps of a lane quarter deal out the chunks of ALL the CTA's tiles in turn: where the chunks of a tile are no multiple of
        // the warps (3 chunks on 2 warps), the odd one of the next tile goes to the warp that had less to do (342 -> 78 80x54 x127:
        // 51.1 -> 44.1 us, 43 -> 25 35x31 x108: 8.0 -> 6.5).
        int ci = sub;  // this warp's next chunk, counted from the current tile's first
        pdl_wait();  // the outputs written below may still be read by the previous kernel
        for (int m = m_first; m < P.m_tiles; m += m_step, ++tile_i, ci -= n_chunks) {
            if (ci >= n_chunks || q * 32 >= tile_rows) continue;
            const uint32_t buf = tile_i & acc_mask, use = tile_i >> acc_shift;
            // which output pixel this thread's TMEM lane holds
            long pix;  // linear (img, oy, ox) index
            long img = 0, inimg = 0;
            bool valid;
            if (P.flat) {
                pix = (long)m * tile_rows + row;
                valid = pix < total_pix && row < tile_rows;
                if (writes(DT_F32_NCHW) || (writes(DT_S8_NHWC) && mixed.out_f32 != nullptr)) {
                    if (total_pix <= 0x7FFFFFFFl) {
                        const uint32_t q32 = fast_div((uint32_t)pix, P.div_plane);
                        img = (long)q32;
                        inimg = pix - (long)q32 * plane;
                    } else {
                        img = pix / plane;
                        inimg = pix - img * plane;
                    }
                }
            } else {
                const int im = (int)fast_div((uint32_t)m, P.div_img);
                const int r = m - im * P.tiles_x * P.tiles_y, ty = (int)fast_div((uint32_t)r, P.div_tx);
                const int oy = ty * P.th + row_y, ox = (r - ty * P.tiles_x) * P.tw + row_x;
                valid = oy < s.oh && ox < s.ow;
                img = im;
                inimg = (long)oy * s.ow + ox;
                pix = img * plane + inimg;
            }
            const uint32_t taddr = tmem_base + buf * (uint32_t)P.acc_stride + ((uint32_t)(q * 32) << 16);
            int8_t* out_s8 = reinterpret_cast<int8_t*>(out) + pix * s.cout_pad + c_base;
            int32_t* out_s32 = reinterpret_cast<int32_t*>(out) + pix * s.cout_pad + c_base;
            float* out_f32 = nullptr;
            if (writes(DT_F32_NCHW)) {
                out_f32 = reinterpret_cast<float*>(out) + (img * s.cout + c_base) * plane + inimg;
            } else if (writes(DT_S8_NHWC) && mixed.out_f32 != nullptr) {
                out_f32 = mixed.plane_of_col != nullptr ? mixed.out_f32 + img * mixed.f32_planes * plane + inimg  // plane chosen per column below
                                                        : mixed.out_f32 + (img * s.cout + c_base) * plane + inimg;
            }
            // 16 accumulator columns -> 16 outputs of this thread's pixel. int8 results come back as 4 packed words in wds
            // (the caller stores them); the other output kinds are stored here.
            auto emit16 = [&](const int (&v)[16], int col0, uint32_t (&wds)[4]) {
                const int c0 = c_base + col0;  // first global output channel of this chunk
                if (writes(DT_S32_NHWC)) {
                    int4* o = reinterpret_cast<int4*>(out_s32 + col0);
#pragma unroll
                    for (int g = 0; g < 4; ++g) o[g] = make_int4(v[g * 4], v[g * 4 + 1], v[g * 4 + 2], v[g * 4 + 3]);
                    return;
                }
                // two fp32 lanes per instruction (fma.rn.f32x2 and friends): each lane rounds exactly like the scalar form
                float y[16];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const float4 si = *reinterpret_cast<const float4*>(s_si + col0 + g * 4);
                    const float4 bi = *reinterpret_cast<const float4*>(s_bi + col0 + g * 4);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const float2 a = make_float2(__int2float_rn(v[g * 4 + 2 * h]), __int2float_rn(v[g * 4 + 2 * h + 1]));
                        const float2 s2 = h ? make_float2(si.z, si.w) : make_float2(si.x, si.y);
                        const float2 b2 = h ? make_float2(bi.z, bi.w) : make_float2(bi.x, bi.y);
                        const float2 t = __ffma2_rn(a, s2, b2);
                        y[g * 4 + 2 * h] = activate_t<ACT>(t.x, ep.act_param0);
                        y[g * 4 + 2 * h + 1] = activate_t<ACT>(t.y, ep.act_param0);
                    }
                }
                if (ACT == kAnyAct) {  // (activate_t<kAnyAct> left the values as they are)
                    if (ep.act_type == ACT_LRELU) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) y[j] = activate_t<ACT_LRELU>(y[j], ep.act_param0);
                    } else if (ep.act_type != ACT_NONE) {
                        const float top = ep.act_type == ACT_RELU6 ? 6.f : __int_as_float(0x7F800000);
#pragma unroll
                        for (int j = 0; j < 16; ++j) y[j] = fminf(activate_t<ACT_RELU>(y[j], 0.f), top);
                    }
                }
                if (writes(DT_F32_NCHW)) {
                    // one plane further per channel: a pointer that walks, and one bounds test per chunk where the chunk is whole
                    float* o = out_f32 + (long)col0 * plane;
                    if (c0 + 16 <= s.cout) {
#pragma unroll
                        for (int j = 0; j < 16; ++j, o += plane) *o = y[j];
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j, o += plane)
                            if (c0 + j < s.cout) *o = y[j];
                    }
                } else {
                    if (out_f32 != nullptr) {
                        // channels that some reader wants in fp32: the planes an fp32-output layer would have written
                        const uint32_t m = (mixed.mask[(c0 >> 5) & 31] >> (c0 & 31)) & 0xFFFFu;
                        if (m != 0u) {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if ((m >> j) & 1u) {
                                    const long pl = mixed.plane_of_col != nullptr ? (long)mixed.plane_of_col[c0 + j] : (long)(col0 + j);
                                    out_f32[pl * plane] = ACT == ACT_POS ? activate(y[j], ep.act_type, ep.act_param0) : y[j];
                                }
                        }
                    }
#pragma unroll
                    for (int g = 0; g < 4; ++g) {
                        float4 so;
                        if constexpr (ONE_SCALE) so = make_float4(ep.scale_out0, ep.scale_out0, ep.scale_out0, ep.scale_out0);
                        else so = *reinterpret_cast<const float4*>(s_so + col0 + g * 4);
                        const float2 ya = make_float2(y[g * 4], y[g * 4 + 1]), yb = make_float2(y[g * 4 + 2], y[g * 4 + 3]), sa = make_float2(so.x, so.y),
                                     sb = make_float2(so.z, so.w);
                        if constexpr (ACT == ACT_POS) {
                            wds[g] = requant4_pos(ya, sa, yb, sb);
                        } else {
                            const int2 qa = round2(__fmul2_rn(ya, sa), half), qb = round2(__fmul2_rn(yb, sb), half);  // (signed: a scale may be negative)
                            wds[g] = pack_sat_s8x4(qa.x, qa.y, qb.x, qb.y);
                        }
                    }
                }
            };
            // Chunks of 32 columns: two TMEM loads in flight, and int8 rows leave as one 32-byte store per thread, a whole
            // DRAM sector (two 16-byte stores from different warps would each touch half of it).
            const bool wide_ok = writes(DT_S8_NHWC) && ((s.cout_pad | (c_base)) & 31) == 0;
            if (!mbar_wait_warp(bar_tfull + 8u * buf, use & 1u, abort_flag, status, 8u, P.wait_ns)) break;
            tc_fence_after();
            for (; ci < n_chunks; ci += nsub) {
                const int col0 = ci * chunk;
                int v[16], v2[16];
                uint32_t wa[4], wb[4];
                const bool two = chunk == 32 && col0 + 16 < P.bn;
                const bool a_ok = c_base + col0 < s.cout_pad, b_ok = two && c_base + col0 + 16 < s.cout_pad;
                __syncwarp();  // tcgen05.ld is warp-collective
                tmem_ld16(taddr + (uint32_t)col0, v);
                if (two) tmem_ld16(taddr + (uint32_t)(col0 + 16), v2);
                tmem_wait_ld16(v);
                tmem_wait_ld16(v2);
                // the chunk is read: its columns may be overwritten from here on
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_tempty + 8u * buf);
                if (valid && a_ok) emit16(v, col0, wa);
                if (valid && b_ok) emit16(v2, col0 + 16, wb);
                if (!valid) continue;
                if (writes(DT_S8_NHWC) && mixed.n_chunks > 0) {
                    // scattered output: each 16-column chunk has its own destination tensor
                    const int ch = (c_base + col0) >> 4;
                    int8_t* da = a_ok ? mixed.dst[ch] : nullptr;
                    int8_t* db = b_ok ? mixed.dst[ch + 1] : nullptr;
                    if (da != nullptr && db != nullptr && ((mixed.pair_ok >> (ch >> 1)) & 1ull) != 0ull && (ch & 1) == 0) {
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(da + pix * mixed.pitch[ch]), "r"(wa[0]),
                                     "r"(wa[1]), "r"(wa[2]), "r"(wa[3]), "r"(wb[0]), "r"(wb[1]), "r"(wb[2]), "r"(wb[3])
                                     : "memory");
                    } else {
                        if (da != nullptr) *reinterpret_cast<uint4*>(da + pix * mixed.pitch[ch]) = make_uint4(wa[0], wa[1], wa[2], wa[3]);
                        if (db != nullptr) *reinterpret_cast<uint4*>(db + pix * mixed.pitch[ch + 1]) = make_uint4(wb[0], wb[1], wb[2], wb[3]);
                    }
                } else if (writes(DT_S8_NHWC)) {
                    if (a_ok && b_ok && wide_ok) {
                        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out_s8 + col0), "r"(wa[0]), "r"(wa[1]),
                                     "r"(wa[2]), "r"(wa[3]), "r"(wb[0]), "r"(wb[1]), "r"(wb[2]), "r"(wb[3])
                                     : "memory");
                    } else {
                        if (a_ok) *reinterpret_cast<uint4*>(out_s8 + col0) = make_uint4(wa[0], wa[1], wa[2], wa[3]);
                        if (b_ok) *reinterpret_cast<uint4*>(out_s8 + col0 + 16) = make_uint4(wb[0], wb[1], wb[2], wb[3]);
                    }
                }
            }
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
    // initialised once, by whichever host thread comes first (function-local statics are thread-safe)
    static const EncodeTiledFn fn = []() -> EncodeTiledFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiledFn>(p);
        return nullptr;
    }();
    return fn;
}

CUtensorMapSwizzle swizzle_for(int bkc) {
    return bkc == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (bkc == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

template <int OUT, int ACT, int BUILD, typename Source, typename Dest>
const char* launch_variant(cudaStream_t stream, int sm_count, const Source& maps, const CUtensorMap& tmB, const UmmaPlan& p,
                           const ConvShape& s, const EpilogueParams& ep, void* out, uint32_t* status, const Dest& mixed) {
    // per-device, per-instantiation set-up; several host threads may drive different GPUs through this function at once
    static std::mutex mu;
    static bool attr_set[64] = {};
    static int regs_per_thread[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    auto kernel = dense_umma_kernel<OUT, ACT, BUILD>;
    int regs = 128;
    if (dev >= 0 && dev < 64) {
        std::lock_guard<std::mutex> lock(mu);
        if (!attr_set[dev]) {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
                return "cudaFuncSetAttribute(MaxDynamicSharedMemorySize) failed";
            cudaFuncAttributes fa{};
            regs_per_thread[dev] = cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs > 0 ? fa.numRegs : 128;
            attr_set[dev] = true;
        }
        regs = regs_per_thread[dev];
    }
    // Tiles are dealt statically to the CTAs of the grid, so a grid larger than what is resident at once runs in waves.
    // The plan bounds residency by shared memory and TMEM; registers and threads are bounded here.
    const int threads = BUILD == kRowsQuantBuild ? build_threads(BUILD) : 64 + 32 * (p.epi_warps + (build_quantizes(BUILD) ? kQuantWarps : 0) + (build_rows(BUILD) ? 1 : 0));
    const int regs_per_warp = (regs * 32 + 255) / 256 * 256;
    int resident = 65536 / (regs_per_warp * (threads / 32));
    if (resident > 2048 / threads) resident = 2048 / threads;
    if (resident < 1) resident = 1;
    const int per_sm = resident < p.ctas_per_sm ? resident : p.ctas_per_sm;
    int per_n = sm_count * per_sm / p.n_tiles;
    if (per_n < 1) per_n = 1;
    if (per_n > p.m_tiles) per_n = p.m_tiles;
    const int grid = per_n * p.n_tiles;
    // the compact plan holds one accumulator: a CTA with a second tile would compute it in columns that are not its own
    if (p.compact && per_n < p.m_tiles) return "compact launch of more than one tile per CTA";
    if (launch_overlapped(kernel, dim3(grid), dim3(threads), (size_t)p.smem_bytes, stream, maps, tmB, p, s, ep, out, status, mixed) != cudaSuccess)
        return "dense_umma_kernel launch failed";
    return nullptr;
}

}  // namespace

static int round_up(int a, int b) { return (a + b - 1) / b * b; }

// What follows from the width of the weight panel (p.bn, p.n_tiles): pipeline depth, tensor memory, shared memory, CTAs per SM.
static bool plan_panel(UmmaPlan& p, int smem_budget) {
    const bool whole = p.gather_whole != 0;
    const long a_stage = p.a_stage_bytes, k_total = p.k_total;
    const long left = (long)smem_budget - 1024 /*alignment slack*/ - 4096 /*barriers + epilogue parameters*/ - (long)p.bn * k_total;
    p.stages = (int)(left / a_stage);
    if (p.stages > 8) p.stages = 8;
    // Small layers (few k-blocks, narrow panels) are latency-bound with one CTA per SM: keep the pipeline short so that
    // several CTAs fit an SM and overlap each other's TMA / MMA / epilogue latencies.
    if ((p.nkb <= 2 || whole) && p.stages > 4) p.stages = 4;
    if (whole && p.stages > 2) p.stages = 2;  // two whole tiles in flight, and room for a second CTA on the SM
    // a halo stage feeds all the taps of a whole pixel tile and channel block: three are a deep enough pipeline
    if (p.halo && p.stages > 3) p.stages = 3;
    if (p.stages < 2) return false;
    // accumulators of bn columns each; TMEM allocations are powers of two >= 32 columns
    p.acc_stride = p.bn <= 32 ? 32 : (p.bn <= 64 ? 64 : (p.bn <= 128 ? 128 : 256));
    // narrow tiles finish quickly; four accumulators let the MMA issuer run three tiles ahead of the epilogue
    p.acc_bufs = p.acc_stride <= 64 ? 4 : 2;
    p.tmem_cols = p.acc_bufs * p.acc_stride;
    // instruction descriptor: D=s32 (2<<4), A=B=signed int8 (1<<7, 1<<10), both K-major, N>>3 at bit 17, M>>4 at bit 24
    p.idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.bn >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
    SmemLayout L = smem_layout(p);
    p.smem_bytes = (int)L.total + 1024;
    // CTAs per SM: TMEM has 512 columns per SM and the hardware scheduler does not account for them, so the shared-memory
    // request is padded until no more CTAs fit an SM than TMEM can serve (a CTA that cannot get its columns would wait
    // inside tcgen05.alloc for a neighbour to finish).
    // eight epilogue warps, two per TMEM lane quarter (sixteen for wide single-CTA tiles, below)
    p.epi_warps = 8;
    int by_tmem = 512 / p.tmem_cols;
    int by_smem = smem_budget / p.smem_bytes;
    p.ctas_per_sm = by_tmem < by_smem ? by_tmem : by_smem;
    if (p.ctas_per_sm > 4) p.ctas_per_sm = 4;
    if (p.ctas_per_sm < 1) p.ctas_per_sm = 1;
    // Wide tiles with one CTA per SM: sixteen epilogue warps (four per lane quarter, 576 threads, the build without a register
    // cap). Requantizing a 128 x 256 tile costs the CUDA cores as much as its MMAs cost the tensor pipe, and eight warps reach
    // only two thirds of the SM's requantize rate (measured: 512 -> 1024: 1660 -> 1837 TOP/s; 256 -> 512: 881 -> 1025; with
    // 128-column tiles it loses, 3x3 128 -> 128: 1938 -> 1865).
    if (p.ctas_per_sm == 1 && p.bn > 128) p.epi_warps = 16;
    const int min_smem = smem_budget / (p.ctas_per_sm + 1) + 1;
    if (p.smem_bytes < min_smem) p.smem_bytes = min_smem;
    return true;
}

static bool plan_layer(int cin, int cout, int kh, int kw, int sh, int sw, int dh, int dw, int smem_budget, UmmaPlan* plan, int bkc_override,
                       bool whole_tile_stages, bool parity_halo) {
    UmmaPlan p{};
    const int cin_pad = nhwc_channels(cin), cout_pad = nhwc_channels(cout);
    if (sh < 1 || sw < 1 || sh > 4 || sw > 4) return false;
    if (cin_pad < 32) return false;        // a TMA box may not be wider than the tensor
    p.bkc = cin_pad >= 128 ? 128 : (cin_pad >= 64 ? 64 : 32);
    if (bkc_override == 32 || bkc_override == 64 || bkc_override == 128) p.bkc = bkc_override;
    p.ncb = (cin_pad + p.bkc - 1) / p.bkc;
    p.taps = kh * kw;
    p.nkb = p.taps * p.ncb;
    const long k_total = (long)p.nkb * p.bkc;
    // largest BN (multiple of 16, <= 256) whose weight panel leaves room for at least 3 A stages,
    // preferring a split of cout_pad into equal tiles
    // strided and dilated layers load one box per filter tap (a strided layer's box takes every sw-th / sh-th pixel: TMA
    // element strides); undilated stride-1 k x k layers load one halo tile per pixel tile
    p.halo = parity_halo ? 2 : (p.taps > 1 && dh == 1 && dw == 1 && sh == 1 && sw == 1) ? 1 : 0;
    const bool whole = whole_tile_stages && !p.halo && p.taps == 1;
    p.gather_whole = whole ? 1 : 0;
    const long a_stage = p.halo == 2 ? (long)ParityHalo(kh, kw).stage_bytes(p.bkc)
                         : p.halo ? ((long)p.bkc * (kHaloTw + kw - 1) * (kHaloTh + kh - 1) + 1023) / 1024 * 1024
                                : (long)kTileM * p.bkc * (whole ? p.nkb : 1);
    p.a_stage_bytes = (int)a_stage;
    const long avail = (long)smem_budget - 1024 /*alignment slack*/ - 4096 /*barriers + epilogue parameters*/ - (whole ? 2 : 3) * a_stage;
    if (avail <= 0) return false;
    long bn_max = avail / k_total;
    bn_max = bn_max > 256 ? 256 : bn_max;
    bn_max = bn_max / 16 * 16;
    if (bn_max < 16) return false;
    p.n_tiles = (cout_pad + (int)bn_max - 1) / (int)bn_max;
    p.bn = round_up((cout_pad + p.n_tiles - 1) / p.n_tiles, 16);
    if (p.bkc == 32) p.bn = round_up(p.bn, 32);  // keeps every weight tile on a 1 KiB boundary
    if (p.bn > 256 || (long)p.bn * k_total > avail) return false;
    p.k_total = (int)k_total;
    p.cout_rows = p.n_tiles * p.bn;
    if (!plan_panel(p, smem_budget)) return false;
    *plan = p;
    return true;
}

bool umma_plan_layer(int cin, int cout, int kh, int kw, int sh, int sw, int dh, int dw, int smem_budget, UmmaPlan* plan, int bkc_override,
                     bool whole_tile_stages) {
    return plan_layer(cin, cout, kh, kw, sh, sw, dh, dw, smem_budget, plan, bkc_override, whole_tile_stages, false);
}

bool umma_plan_parity(const UmmaPlan& taps, int cin, int cout, int kh, int kw, int sh, int sw, int dh, int dw, int smem_budget, UmmaPlan* plan) {
    return sh == 2 && sw == 2 && dh == 1 && dw == 1 && kh > 1 && kw > 1 && kh <= 7 && kw <= 7 &&
           plan_layer(cin, cout, kh, kw, sh, sw, dh, dw, smem_budget, plan, taps.bkc > 64 ? 64 : 0, false, true) && plan->n_tiles <= taps.n_tiles;
}

bool umma_narrow_plan(const UmmaPlan& base, int bn, int cout, int smem_budget, UmmaPlan* plan) {
    UmmaPlan p = base;
    p.bn = bn;
    p.n_tiles = (nhwc_channels(cout) + bn - 1) / bn;
    if (bn >= base.bn || p.n_tiles <= base.n_tiles || !plan_panel(p, smem_budget)) return false;
    *plan = p;
    return true;
}

std::vector<UmmaVariant> umma_variants(const UmmaPlan& widest, int cout, int smem_budget) {
    std::vector<UmmaVariant> all(1);
    all[0].plan = widest;
    UmmaVariant v;
    for (int bn : {128, 64, 32})
        if (umma_narrow_plan(widest, bn, cout, smem_budget, &v.plan)) all.push_back(v);
    return all;
}

// What follows from a plan's panel, tile and team shape with channels as accumulator rows: pipeline, tensor memory, CTAs per SM.
static bool plan_rows(UmmaPlan& p, int cout_pad, int smem_budget) {
    const bool quant = p.rows == rows_pixels(kRowsQuantBuild);
    p.n_tiles = (cout_pad + p.bn - 1) / p.bn;
    p.acc_stride = p.rows;
    p.idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.rows >> 3) << 17) | ((uint32_t)(kTileM >> 4) << 24);
    // Two CTAs per SM of eight epilogue warps and two accumulators each, or one of sixteen and four: the same warps and tensor memory,
    // but two panels, and while one CTA's warps wait for an accumulator the other's have one.
    p.epi_warps = 8;
    p.stages = 1;
    p.out_slots = 2;
    p.boxes = quant ? kBoxWarps : 0;
    int fixed = (int)smem_layout(p).total - p.a_stage_bytes + 1024;
    auto stages_in = [&](int budget) { return budget > fixed ? (budget - fixed - 512 /*barriers of further stages and boxes*/) / p.a_stage_bytes : 0; };
    const int most = quant ? 8 : p.gather_whole ? 2 : p.nkb <= 2 ? 4 : 8;
    const bool pair = !quant && p.bn <= kTileM && stages_in(smem_budget / 2) >= 2;
    p.ctas_per_sm = pair ? 2 : 1;
    p.stages = stages_in(smem_budget / p.ctas_per_sm);
    // two finished tiles per team, if three (of a tile in several loads: four) stages remain
    if (!quant && !pair && stages_in(smem_budget - 2 * (int)out_slot_bytes(p)) >= (p.nkb > 1 && !p.gather_whole ? 4 : 3)) {
        p.out_slots = kOutSlots;
        fixed += 2 * (int)out_slot_bytes(p);
        p.stages = stages_in(smem_budget);
    }
    // twice as many boxes and finished tiles, if stages for as many tiles as the warps have boxes of, and one more, remain
    const int want = quant ? kBoxWarps / (p.k_total / kBoxChannels) + 2 : 0;
    if (quant && stages_in(smem_budget - kBoxWarps * (int)kBoxBytes) >= want) {
        p.boxes = 2 * kBoxWarps;
        fixed += kBoxWarps * (int)kBoxBytes;
    }
    if (quant && stages_in(smem_budget - 2 * (int)out_slot_bytes(p)) >= want) {
        p.out_slots = kOutSlots;
        fixed += 2 * (int)out_slot_bytes(p);
    }
    if (quant) p.stages = stages_in(smem_budget);
    if (p.stages > most) p.stages = most;
    if (p.stages < 2) return false;
    p.acc_bufs = quant ? 8 : pair ? 2 : 4;
    p.tmem_cols = p.acc_bufs * p.acc_stride;
    if (!quant && !pair) p.epi_warps = 16;
    p.smem_bytes = (int)smem_layout(p).total + 1024;
    const int min_smem = smem_budget / (p.ctas_per_sm + 1) + 1;  // (no more CTAs than tensor memory serves, see plan_panel)
    if (p.smem_bytes < min_smem) p.smem_bytes = min_smem;
    return true;
}

std::vector<UmmaVariant> umma_row_variants(const UmmaPlan& base, int cout, int smem_budget) {
    std::vector<UmmaVariant> all;
    const int cout_pad = nhwc_channels(cout);
    if (base.taps != 1) return all;
    for (int bn : {256, 192, 128, 64}) {
        if (bn >= cout_pad + 64 || (bn == 64 && cout_pad > 64)) continue;
        UmmaVariant v;
        v.plan = base;
        v.plan.rows = rows_pixels(kRowsBuild);
        v.plan.bn = v.plan.panel_box = bn;
        if (plan_rows(v.plan, cout_pad, smem_budget)) all.push_back(v);
    }
    // fp32 input, quantized inside: one panel of all the channels, so that the input is quantized once; a stage holds a whole tile
    UmmaVariant v;
    v.plan = base;
    v.plan.rows = rows_pixels(kRowsQuantBuild);
    v.plan.bn = round_up(cout_pad, 64);
    v.plan.panel_box = 64;
    v.plan.a_stage_bytes = v.plan.rows * base.k_total;
    if (!base.gather && v.plan.bn <= kRowsMaxBlocks * kTileM && plan_rows(v.plan, cout_pad, smem_budget)) all.push_back(v);
    return all;
}

void umma_pack_weights(const UmmaPlan& p, const int8_t* w_oihw, int cin, int cout, int kh, int kw, int8_t* dst) {
    // dst[cout_rows][k_total], k = (tap*ncb + cb)*bkc + (channel - cb*bkc); zero elsewhere
    const long kt = p.k_total;
    for (long i = 0; i < (long)p.cout_rows * kt; ++i) dst[i] = 0;
    for (int o = 0; o < cout; ++o)
        for (int c = 0; c < cin; ++c)
            for (int t = 0; t < kh * kw; ++t) {
                const int cb = c / p.bkc, ci = c % p.bkc;
                dst[o * kt + ((long)t * p.ncb + cb) * p.bkc + ci] = w_oihw[((long)o * cin + c) * kh * kw + t];
            }
}

const char* umma_encode_weight_map(const UmmaPlan& p, const int8_t* w_dev, void* map_out) {
    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return "cuTensorMapEncodeTiled entry point not available";
    cuuint64_t dims[2] = {(cuuint64_t)p.k_total, (cuuint64_t)p.cout_rows};
    cuuint64_t strides[1] = {(cuuint64_t)p.k_total};
    cuuint32_t box[2] = {(cuuint32_t)p.bkc, (cuuint32_t)(p.rows ? p.panel_box : p.bn)};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(reinterpret_cast<CUtensorMap*>(map_out), CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)w_dev, dims, strides, box,
                     estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle_for(p.bkc), CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? nullptr : "cuTensorMapEncodeTiled(weights) failed";
}

bool umma_box_input(const UmmaFloatInput& in, long hw) {
    return in.n_runs == 1 && hw % 4 == 0 && (reinterpret_cast<uintptr_t>(in.base[0]) & 15) == 0 && in.img_stride[0] % 4 == 0;
}

// Describes an fp32 input for quantization inside the kernel; false when its planes are scattered over more runs than that takes.
bool umma_float_input(const float* x, const PlaneGather* table, int cin, long hw, float scale, UmmaFloatInput* in) {
    in->scale = scale;
    in->n_runs = 0;
    if (!table) {
        in->base[0] = x;
        in->img_stride[0] = (long long)cin * hw;
        in->first[0] = 0;
        in->n_runs = 1;
        return true;
    }
    for (int c = 0; c < cin; ++c) {
        if (c > 0 && table->ref[c] == table->ref[c - 1] + 1) continue;
        if (in->n_runs == kQuantRuns) return false;
        const int b = (int)(table->ref[c] >> 24);
        in->base[in->n_runs] = table->base[b] + (long long)(table->ref[c] & 0xFFFFFFu) * hw;
        in->img_stride[in->n_runs] = table->img_stride[b];
        in->first[in->n_runs++] = c;
    }
    return true;
}

namespace {

// How a plan tiles the output pixels of a call.
struct PixelTiles {
    int flat, tw, th, x, y;
    long tiles;
};
PixelTiles tile_pixels(const UmmaPlan& p, const ConvShape& s) {
    PixelTiles t{};
    t.flat = s.kh == 1 && s.kw == 1 && s.ph == 0 && s.pw == 0 && s.sh == 1 && s.sw == 1 ? 1 : 0;
    if (t.flat) {
        t.tw = kTileM; t.th = 1; t.y = 1;
        t.tiles = ((long)s.n * s.oh * s.ow + kTileM - 1) / kTileM;
        t.x = (int)t.tiles;
        return t;
    }
    // rectangle of 128 output pixels with the least padding waste (halo mode: always 8 x 16)
    long best = -1;
    for (int tw = 8; tw <= 128; tw *= 2) {
        const int th = kTileM / tw;
        if ((tw - 1) * s.sw + 1 > 256 || (th - 1) * s.sh + 1 > 256) continue;  // a TMA box spans at most 256 elements per dimension
        const long cover = (long)((s.ow + tw - 1) / tw) * tw * ((s.oh + th - 1) / th) * th;
        if (best < 0 || cover < best) { best = cover; t.tw = tw; t.th = th; }
    }
    if (p.halo) { t.tw = kHaloTw; t.th = kHaloTh; }
    t.x = (s.ow + t.tw - 1) / t.tw;
    t.y = (s.oh + t.th - 1) / t.th;
    t.tiles = (long)s.n * t.x * t.y;
    return t;
}

// Width of the weight panels. A launch with fewer CTAs than SMs is bound by the chain of one tile, most of which (MMAs, requantize,
// stores) shrinks with the panel, so panels of 128 and 64 columns are taken as long as all the CTAs are resident at once. Panels of 32
// halve little more than the fixed part of that chain and read the activations twice as often, which other streams pay for: only
// where every CTA still has an SM to itself. A panel that is not a quarter narrower than the next wider one adds a pass and saves
// little: not while half the SMs are free. 1x1, us with the panels the rule takes / wider ones / narrower ones: 96 -> 512, 40 tiles
// 4.8 / 7.8 / 5.5; 196 -> 140, 60 tiles (3 panels) 4.1 / 4.9 / 4.7; 205 -> 56, 133 tiles (1) 4.3 / - / 4.4; over 500 layers of 24 to 1024
// channels 1.1 % from the best of every layer. Three ShuffleNetV2 forwards at a time, 9 images each: 122 us a forward, with panels of
// 32 wherever they are resident 141.
// A k x k layer's panel holds all its taps. Where two CTAs do not fit an SM for it, the next launch's panels come in beside this
// one's only if half the SMs are free (202 -> 130 3x3 10x15 x12: 72 CTAs 5.3, 120 narrower ones 6.8).
constexpr int kNarrowPanel = 32;
int pick_panels(const UmmaVariant* v, int n, long tiles, int sm_count) {
    int pick = 0;
    for (int i = 1; i < n && tiles * v[pick].plan.n_tiles < sm_count; ++i) {
        const UmmaPlan& p = v[i].plan;
        if (4 * p.bn > 3 * v[pick].plan.bn && 2 * tiles * v[pick].plan.n_tiles <= sm_count) continue;
        const long room = p.halo && p.ctas_per_sm == 1 ? sm_count / 2 : (long)sm_count * (p.bn <= kNarrowPanel ? 1 : p.ctas_per_sm);
        if (tiles * p.n_tiles <= room) pick = i;
    }
    return pick;
}

// Pixels per tile of a one-tile-per-CTA launch. SMs still idle: fewer. A tile's loads arrive a row at a time, and a gathered layer has a row of
// 32 bytes per pixel and K block (232 channels gathered in 15 blocks: 1900 rows for 128 pixels). 128 / 64 / 32 / 16 pixels at most: 116 -> 116
// 20x20 2.59 / 2.47 / 2.37 / 2.30 us, detector on one 416x416 image 450 / 433 / 429 / 427, backbone 169 / 164 / 160 / 159. A quantizing
// launch, whose CTAs have an SM to themselves, keeps 32 (116 -> 116: 3.8, with 16 4.4).
int small_tile_rows(long pixels, int n_tiles, bool inside, int sm_count) {
    int rows = kTileM;
    while (rows > (inside ? 32 : 16) && (pixels + rows / 2 - 1) / (rows / 2) * n_tiles <= sm_count) rows /= 2;
    return rows;
}

// Whether a launch of one tile per CTA runs the compact build. A quantizing one always does; on int8 input a halo tile wants its MMA issue
// unrolled (rolled it costs 0.9 us), and a wide panel the unrolled epilogue (compact / specialised, 130 layers alone: 32 columns 0.97,
// 64 1.04, 128 1.11, 240 1.21; in a chain of layers the compact build gains what kAnyOut says).
bool runs_compact(const UmmaPlan& p, long tiles, bool inside, int sm_count) {
    return tiles * p.n_tiles <= sm_count && (inside || (!p.halo && p.bn <= 64));
}

// Costs (us) of a flat launch on fp32 input: quantized inside, one tile per CTA, and through an int8 copy. Fitted to 250 layers of 33 to 1024
// channels (7 and 9 % from the measured times): the eight quantizing warps' items, the operand bytes of a tile, the panel's columns
// and bytes; the quantize kernel and what the convolution behind it takes.
double inside_us(const UmmaPlan& p, const ConvShape& s, int rows) {
    const bool quads = (long)s.h * s.w % 4 == 0;
    const double items = (quads ? (rows + 127) / 128 : (rows + 31) / 32) * (p.k_total / 16) / (double)kQuantWarps;
    return 2.9 + (quads ? 0.79 : 0.42) * items + 3.5e-5 * rows * p.k_total + 0.012 * p.bn + 2.8e-6 * p.bn * p.k_total + 6.7e-4 * p.k_total;
}
double copy_us(const UmmaPlan& p, const ConvShape& s, long tiles, int sm_count) {
    const double per_sm = (double)((tiles * p.n_tiles + sm_count - 1) / sm_count);
    return 4.9 + 8.1e-7 * s.n * s.h * s.w * s.cin_pad + 2.1e-3 * p.k_total + 1.6e-3 * p.bn + per_sm * (9.6e-3 * p.bn + 6e-4 * p.k_total);
}

}  // namespace

// Stride 2: the two parity planes of a tile's halo are half the rows of one box per tap (3x3: 561 against 1152; us: 64 -> 128 75x75 x32,
// fp32 out 14.1 -> 11.8, int8 out 13.5 -> 10.4; 173 -> 93 57x20 x44 22.1 -> 13.6; 40 -> 40 40x40 x64 12.3 -> 8.7; 64 -> 64 56x56 one image
// 4.6 -> 3.8), but its tiles are 8 x 16 whatever the map is, while the other form takes the rectangle that covers it best. Where
// that makes half as many tiles again, and not all of them run at once, the advantage is gone: 53 -> 44 9x59 x101, 404 tiles against
// 202, 8.1 / 6.0; 32 -> 32 8x40 x128, 384 against 128, 6.2 / 4.7; 154 -> 140 13x32 x78, 156 against 78, 16.9 / 14.2 (250 layers: 0.5 %
// from the better form of each on average; always by parity 0.9 %, always by tap 22 %).
bool umma_prefers_parity(const UmmaVariant* parity, int n_parity, const UmmaVariant* taps, const ConvShape& s, int sm_count) {
    const long by_parity = tile_pixels(parity[0].plan, s).tiles, by_tap = tile_pixels(taps[0].plan, s).tiles;
    return 2 * by_parity <= 3 * by_tap || by_parity * parity[pick_panels(parity, n_parity, by_parity, sm_count)].plan.n_tiles <= sm_count;
}

// fp32 input, 1x1: inside where that is estimated to be faster, over the panels for which it is fastest (every panel quantizes the input once
// more, but a narrower one may leave the launch short tiles). 196 -> 140 48x31 x5: 59 tiles, one panel 7.3 us; three of 64 columns, two
// tiles for some CTAs, 8.6; through a copy 8.3. With more tiles than SMs one panel that does not want sixteen
// epilogue warps wins, where the images are whole pixel quads (116 -> 116 20x20 x256: copy / inside 17.5 / 16.1; but two panels,
// 256 -> 512 28x28 x128: 52 / 55, and pixel by pixel, 90 -> 77 31x33 x60: 12.5 / 19.2). Halo tiles: up to 64 channels in one block and one
// wave of CTAs, panels narrowed into half of one (64 -> 64 56x56 one image 8.5 / 5.3; 128 -> 128 28x28 x8 8.8 / 11.6).
UmmaChoice umma_choose(const UmmaVariant* v, int n, const ConvShape& s, int sm_count, bool may_quantize, long* n_tiles) {
    const PixelTiles t = tile_pixels(v[0].plan, s);
    if (n_tiles) *n_tiles = t.tiles;
    const long pixels = (long)s.n * s.oh * s.ow;
    UmmaChoice c{v + pick_panels(v, n, t.tiles, sm_count), false, kTileM, false, false};
    const bool can = may_quantize && (t.flat || v[0].plan.halo == 1) && s.cin_pad > 32 && (double)s.n * s.h * s.w <= 2147483647.0;
    if (can && !t.flat && v[0].plan.ncb == 1 && s.cin_pad <= 64 && t.tiles * v[0].plan.n_tiles <= sm_count) {
        c.variant = v;
        c.inside = true;
        for (int i = 1; i < n; ++i)
            if (2 * t.tiles * v[i].plan.n_tiles <= sm_count) c.variant = v + i;
    } else if (can && t.flat && t.tiles * v[0].plan.n_tiles <= sm_count) {
        double best = copy_us(c.variant->plan, s, t.tiles, sm_count);
        for (int i = 0; i < n && t.tiles * v[i].plan.n_tiles <= sm_count; ++i) {
            const double us = inside_us(v[i].plan, s, small_tile_rows(pixels, v[i].plan.n_tiles, true, sm_count));
            if (us >= best) continue;
            best = us;
            c.variant = v + i;
            c.inside = true;
        }
    } else if (can && t.flat && v[0].plan.n_tiles == 1 && v[0].plan.bn <= 192 && (long)s.h * s.w % 4 == 0) {
        c.variant = v;
        c.inside = true;
    }
    c.compact = runs_compact(c.variant->plan, t.tiles, c.inside, sm_count);
    if (c.compact && t.flat) c.tile_rows = small_tile_rows(pixels, c.variant->plan.n_tiles, c.inside, sm_count);
    return c;
}

// Channels as accumulator rows (builds 6 and 7 of the comment in front of the kernel; 8 below). What they gain is the epilogue; an
// MMA of 128 channels x 128 pixels reads as many bytes of shared memory as its port delivers in the time it takes, one of 128 pixels x
// 256 channels three quarters of them, so with more input channels the order of the operands that keeps the port free is the better one.
// us, pixels as rows / channels as rows: 64 -> 256 56x56 x128 41.8 / 26.0, 256 -> 512 28x28 x128 23.9 / 18.5, 116 -> 116 20x20 x256 9.3 / 6.5,
// 58 -> 58 40x40 x256 14.2 / 11.0, 512 -> 1024 28x28 x32 17.3 / 15.4; 110 layers of 24 to 1024 channels: up to 256 input channels 1.0 to 1.45
// times as fast, 512 and 64 or whole panels of 256 output channels 1.05 to 1.15, else slower (323 -> 387, 369 tiles 14.2 / 21.9; 587 -> 86, 556
// tiles 9.8 / 11.6). An accumulator is 128 or 64 channels, and what a layer does not fill is computed all the same: up to two fifths
// more (73 -> 87, 1608 tiles 13.6 / 12.2; but 43 -> 25, 916 tiles 6.3 / 6.8). The panel that wastes least; among equals the widest, which fetches
// the pixels fewest times (256 -> 512: 256 channels 18.4, 128 21.1), but up to four rounds of CTAs two small CTAs per SM (112 -> 250, 542
// tiles 8.6 / 8.0; 232 -> 232, 200 tiles 6.5 / 5.9). Small launches keep their narrow panels of pixels. k x k layers read every pixel once per
// tap and are bound by the MMAs: 192 of them 0.77 times as fast.
// fp32 input that a quantize kernel brings: the kernel behind this one is likely another of its kind, and then starts better when this one
// ends than as soon as there is room beside it (us, beside / at the end: 256 -> 512 28x28 x128 54.9 / 44.1, 307 -> 490 102648 pixels 65.9 /
// 54.1, 473 -> 903 29520 pixels 35.1 / 30.9, 116 -> 974 6831 pixels 9.2 / 7.9; of up to 64 channels 45 -> 330 10260 pixels 6.7 / 7.5, 34 -> 473
// 16640 pixels 8.7 / 9.4).
// An fp32 input that fills L2 by itself is quantized inside, where one panel holds all the channels: the int8 copy then goes to HBM and
// back, and the planes can be fetched while other tiles are multiplied. us, other forms / this one: 256 -> 512 28x28 x128 (103 MB) 44.1 /
// 38.7, 249 -> 61 192660 pixels 47.9 / 42.2, 620 -> 37 109800 pixels 59.7 / 54.0; but 105 -> 453 55200 pixels (23 MB) 16.6 / 18.8, 178 -> 58 54880
// pixels (39 MB) 11.6 / 13.5, 120 -> 46 143000 pixels (69 MB) 18.3 / 20.7.
// Its tiles of 64 pixels hold one image each, so that small planes leave them empty (43 -> 263 2x2 x143215 128 / 1773, 122 -> 382 6x4 x12099 66 / 155,
// 170 -> 468 8x6 x4057 69.1 / 78.5): seven eighths full. Of 215 layers of 17 to 1024 channels, 40 to 400 MB, those whose tiles are: with few
// input channels the accumulators are the longer half, and half-empty or many of them lose (92 -> 145 31x100 x359 151 / 181, 66 -> 137 55 / 64, 58 ->
// 505 151 / 192, 83 -> 437 177 / 192; 101 -> 177 57 / 53, 80 -> 50 44.9 / 31.4); up to 384 they gain 1.00 to 1.58; above, the tile's operand and the weights
// leave room for two or three stages, and only one narrow or full accumulators gain (434 -> 37 44.7 / 39.3, 624 -> 115 110 / 92; 511 -> 109 65 / 77, 612 -> 81
// 42 / 51); above 640 none (700 -> 47 85 / 97, 722 -> 51 46.5 / 52.7).
constexpr double kFillsL2 = 96.0 * (1 << 20);
bool box_tiles_pay(const UmmaPlan& p, const ConvShape& s) {
    const long hw = (long)s.h * s.w, in_tiles = (hw + p.rows - 1) / p.rows * p.rows;
    if (4.0 * s.cin * s.n * hw < kFillsL2 || 8 * hw < 7 * in_tiles) return false;
    if (p.k_total <= 128) return p.bn <= kTileM || (p.bn <= 3 * kTileM && 8 * s.cout_pad >= 7 * p.bn);
    return p.k_total <= 384 || (p.k_total <= 640 && (p.bn <= 64 || 8 * s.cout_pad > 7 * p.bn));
}
UmmaChoice umma_choose_rows(const UmmaChoice& choice, const UmmaVariant* rows, int n_rows, const ConvShape& s, int sm_count, bool f32_input, bool may_box) {
    const PixelTiles t = tile_pixels(choice.variant->plan, s);
    if (may_box && !choice.compact && t.flat && (double)s.n * s.h * s.w <= 2147483647.0 && n_rows > 0 &&
        rows[n_rows - 1].plan.rows == rows_pixels(kRowsQuantBuild) && box_tiles_pay(rows[n_rows - 1].plan, s)) {
        UmmaChoice c = choice;
        c.variant = &rows[n_rows - 1];
        c.inside = true;
        c.tile_rows = c.variant->plan.rows;
        return c;
    }
    if (choice.inside || choice.compact || !t.flat || (choice.variant->plan.bn <= 64 && t.tiles <= sm_count)) return choice;
    const UmmaVariant* pick = nullptr;
    int pick_work = 0;
    for (int i = 0; i < n_rows; ++i) {
        const UmmaPlan& p = rows[i].plan;
        if (p.rows != rows_pixels(kRowsBuild)) continue;
        const int widest = s.cout_pad < p.bn ? s.cout_pad : p.bn, work = p.n_tiles * ((widest + 63) / 64);
        const bool light = p.k_total <= 256;
        if (64 * work * (light ? 5 : 7) > s.cout_pad * (light ? 7 : 8)) continue;
        if (p.k_total > 512 || (!light && p.bn % 256 != 0 && p.bn != 64)) continue;
        if (pick && work >= pick_work && !(work == pick_work && light && p.bn == kTileM && t.tiles * pick->plan.n_tiles < 4l * sm_count)) continue;
        pick = &rows[i];
        pick_work = work;
    }
    UmmaChoice c = choice;
    if (pick) {
        c.variant = pick;
        c.late = f32_input && pick->plan.k_total > 64;
    }
    return c;
}

const char* launch_dense_umma(cudaStream_t stream, int sm_count, const UmmaChoice& choice, const ConvShape& s,
                              const int8_t* x, const EpilogueParams& ep, void* out, int out_dtype, uint32_t* status,
                              const UmmaSources* sources, const UmmaMixedOut* mixed_in, unsigned long long wait_limit_ns, const UmmaFloatInput* f32) {
    EncodeTiledFn enc = get_encode_fn();
    if (!enc) return "cuTensorMapEncodeTiled entry point not available";
    const long pixels = (long)s.n * s.oh * s.ow;
    if (pixels == 0) return nullptr;
    if ((f32 != nullptr) != choice.inside) return "fp32 input without a launch that quantizes it (or the reverse)";
    UmmaPlan p = choice.variant->plan;
    const PixelTiles tiles = tile_pixels(p, s);
    p.flat = tiles.flat; p.tw = tiles.tw; p.th = tiles.th; p.tiles_x = tiles.x; p.tiles_y = tiles.y; p.m_tiles = (int)tiles.tiles;
    p.tile_rows = choice.tile_rows;
    p.late = choice.late ? 1 : 0;
    if (p.tile_rows != kTileM) p.m_tiles = p.tiles_x = (int)((pixels + p.tile_rows - 1) / p.tile_rows);
    if (f32 && p.rows) {  // tiles of one image each
        p.tiles_x = (int)(((long)s.h * s.w + p.rows - 1) / p.rows);
        p.m_tiles = s.n * p.tiles_x;
    }
    const bool flat = p.flat != 0;
    KernelMaps km;  // only the entries the plan uses are filled in
    CUtensorMap& tmA = km.tm[0];
    UmmaMixedOut mixed{};
    if (mixed_in) {
        if (out_dtype != DT_S8_NHWC || s.cout > 1024) return "fp32 side output needs an int8 launch with at most 1024 output channels";
        mixed = *mixed_in;
    }
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = CUDA_SUCCESS;
    if ((p.gather > 0) != (sources != nullptr)) return "gathered layer launched without its sources (or the reverse)";
    if (p.gather > 0) {
        if (!flat || sources->n_src != p.gather || p.nkb > kUmmaMaxGatherBlocks || p.bkc != kUmmaGatherBlock) return "bad gathered launch";
        for (int i = 0; i < sources->n_src && r == CUDA_SUCCESS; ++i) {
            const cuuint64_t cp = (cuuint64_t)sources->src_cpad[i];
            cuuint64_t dims[4] = {cp, (cuuint64_t)pixels, 1, 1};
            cuuint64_t strides[3] = {cp, cp * pixels, cp * pixels};
            cuuint32_t box[4] = {(cuuint32_t)p.bkc, (cuuint32_t)p.tile_rows, 1, 1};
            r = enc(&km.tm[i], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)sources->src[i], dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_for(p.bkc), CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        }
        for (int kb = 0; kb < p.nkb; ++kb) {
            km.block_x[kb] = sources->block_x[kb];
            km.block_src[kb] = sources->block_src[kb];
        }
    } else if (flat) {
        cuuint64_t dims[4] = {(cuuint64_t)s.cin_pad, (cuuint64_t)pixels, 1, 1};
        cuuint64_t strides[3] = {(cuuint64_t)s.cin_pad, (cuuint64_t)s.cin_pad * pixels, (cuuint64_t)s.cin_pad * pixels};
        cuuint32_t box[4] = {(cuuint32_t)p.bkc, (cuuint32_t)p.tile_rows, 1, 1};
        if (!f32)
            r = enc(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_for(p.bkc), CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    } else {
        cuuint64_t dims[4] = {(cuuint64_t)s.cin_pad, (cuuint64_t)s.w, (cuuint64_t)s.h, (cuuint64_t)s.n};
        cuuint64_t strides[3] = {(cuuint64_t)s.cin_pad, (cuuint64_t)s.cin_pad * s.w, (cuuint64_t)s.cin_pad * s.w * s.h};
        // a strided layer's box spans (tw - 1) * sw + 1 columns of which the traversal takes every sw-th: tw land in shared memory
        const ParityHalo parity(s.kh, s.kw);
        const int cols = p.halo == 2 ? 2 * parity.cols[0] - 1 : p.halo ? p.tw + s.kw - 1 : (p.tw - 1) * s.sw + 1;
        const int rows = p.halo == 2 ? parity.rows : p.halo ? p.th + s.kh - 1 : (p.th - 1) * s.sh + 1;
        cuuint32_t box[4] = {(cuuint32_t)p.bkc, (cuuint32_t)cols, (cuuint32_t)rows, 1};
        estr[1] = (cuuint32_t)s.sw;
        estr[2] = (cuuint32_t)(p.halo == 2 ? 1 : s.sh);
        if (!f32)
            r = enc(&tmA, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_for(p.bkc), CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (p.halo == 2 && r == CUDA_SUCCESS) {
            box[1] = (cuuint32_t)(2 * parity.cols[1] - 1);
            r = enc(&km.tm[1], CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)x, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_for(p.bkc), CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        }
    }
    if (r != CUDA_SUCCESS) return "cuTensorMapEncodeTiled(activations) failed";
    p.wait_ns = wait_limit_ns;
    p.div_img = make_fast_div((uint32_t)(p.tiles_x * p.tiles_y));
    p.div_tx = make_fast_div((uint32_t)p.tiles_x);
    p.div_plane = make_fast_div((uint32_t)(s.oh * s.ow));

    const CUtensorMap& tmB = *reinterpret_cast<const CUtensorMap*>(choice.variant->weight_map);
    const char* err = nullptr;
    QuantSource qs;
    if (f32) {
        p.epi_warps = kMaxEpiWarps;
        p.ctas_per_sm = 1;
        p.smem_bytes = p.smem_bytes > 116 * 1024 ? p.smem_bytes : 116 * 1024;  // one CTA per SM: tensor memory is budgeted for one
        qs.scale = f32->scale;
        qs.half = half_bits(ep.rounding);
        qs.div_halo = make_fast_div((uint32_t)(kHaloTw + s.kw - 1));
        const long hw = (long)s.h * s.w;
        qs.vec = hw % 4 == 0 ? 1 : 0;
        for (int i = 0; i < kQuantRuns; ++i) {
            const bool used = i < f32->n_runs;
            qs.base[i] = used ? f32->base[i] : nullptr;
            qs.img_stride[i] = used ? f32->img_stride[i] : 0;
            qs.first[i] = used ? f32->first[i] : 1 << 30;
            if (used && ((reinterpret_cast<uintptr_t>(qs.base[i]) & 15) != 0 || qs.img_stride[i] % 4 != 0)) qs.vec = 0;
        }
    }
#define OTT_UMMA_LAUNCH(OUT, ACT)                                                                                     \
    err = f32                 ? launch_variant<OUT, ACT, kQuantBuild>(stream, sm_count, qs, tmB, p, s, ep, out, status, mixed) \
          : p.ctas_per_sm > 1 ? launch_variant<OUT, ACT, 1>(stream, sm_count, km, tmB, p, s, ep, out, status, mixed) \
          : p.epi_warps == 16 ? launch_variant<OUT, ACT, 2>(stream, sm_count, km, tmB, p, s, ep, out, status, mixed) \
                              : launch_variant<OUT, ACT, 0>(stream, sm_count, km, tmB, p, s, ep, out, status, mixed)
#define OTT_UMMA_ACT(OUT)                                \
    switch (ep.act_type) {                               \
        case ACT_RELU: OTT_UMMA_LAUNCH(OUT, ACT_RELU); break;   \
        case ACT_LRELU: OTT_UMMA_LAUNCH(OUT, ACT_LRELU); break; \
        case ACT_RELU6: OTT_UMMA_LAUNCH(OUT, ACT_RELU6); break; \
        default: OTT_UMMA_LAUNCH(OUT, ACT_NONE); break;         \
    }
    // One more build in a chain of small launches is one more kernel whose code the SMs have to fetch (0.45 us per launch over a
    // network on one image, where only some layers have one scale): from 2^25 outputs on the saved loads are worth several times that.
    const bool one_scale = ep.one_scale_out && pixels * s.cout_pad >= (1l << 25);
    // One tile per CTA: the launch is a chain whose longest part is fetching its own code, see kAnyOut (detector on one 416x416 image
    // 488 -> 440 us, backbone on one 320x320 image 180 -> 168). The next launch of such a chain sets itself up meanwhile where there is
    // room for it on the same SMs, so the plan takes no more than one tile needs: eight epilogue warps at 96 registers, the stages of
    // one tile, one accumulator (464 -> 1024 on 10x10, 128 CTAs: 4.6 -> 3.5 us).
    p.out_kind = out_dtype;
    if (choice.compact) {
        p.compact = 1;
        p.epi_warps = kMaxEpiWarps;
        const int loads = p.halo ? p.ncb : (p.gather && p.gather_whole ? 1 : p.nkb);
        if (p.stages > loads) p.stages = loads;
        while (p.stages > 2 && smem_layout(p).total + 1024 > kHalfSm) --p.stages;
        p.smem_bytes = (int)smem_layout(p).total + 1024;
        p.acc_bufs = 2;  // (of which the one tile uses the first)
        p.tmem_cols = p.acc_stride;
        err = f32 ? launch_variant<kAnyOut, kAnyAct, kCompactQuantBuild>(stream, sm_count, qs, tmB, p, s, ep, out, status, mixed)
                  : launch_variant<kAnyOut, kAnyAct, kCompactBuild>(stream, sm_count, km, tmB, p, s, ep, out, status, mixed);
    } else if (p.rows) {
        if (mixed_in || out_dtype != DT_S8_NHWC || !flat) return "a launch with channels as accumulator rows is a 1x1 layer with one int8 output";
        RowsOut to{};
        // which of the two some panel's accumulators want (a map costs the host 0.2 us)
        const int last = s.cout_pad - (p.n_tiles - 1) * p.bn;
        auto ends_in_64 = [](int cols) { return (cols - 1) % kTileM < 64; };
        const bool want_64 = ends_in_64(last) || (p.n_tiles > 1 && ends_in_64(p.bn)), want_128 = last > 64 || (p.n_tiles > 1 && p.bn > 64);
        const cuuint64_t cp = (cuuint64_t)s.cout_pad, hw = (cuuint64_t)s.h * s.w;
        cuuint64_t dims[3] = {cp, f32 ? hw : (cuuint64_t)pixels, f32 ? (cuuint64_t)s.n : 1}, strides[2] = {cp, cp * dims[1]};
        for (int width : {128, 64}) {
            if (!(width == 64 ? want_64 : want_128)) continue;
            cuuint32_t box[3] = {(cuuint32_t)width, (cuuint32_t)p.rows, 1}, one[3] = {1, 1, 1};
            if (enc(width == 128 ? &to.full : &to.half, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, out, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    swizzle_for(width), CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return "cuTensorMapEncodeTiled(output) failed";
        }
        BoxSource planes;
        if (f32) {
            planes.scale = f32->scale;
            planes.half = half_bits(ep.rounding);
            cuuint64_t xd[3] = {hw, (cuuint64_t)s.cin, (cuuint64_t)s.n}, xs[2] = {hw * 4, (cuuint64_t)f32->img_stride[0] * 4};
            cuuint32_t box[3] = {(cuuint32_t)p.rows, (cuuint32_t)kBoxChannels, 1}, one[3] = {1, 1, 1};
            if (f32->n_runs != 1 || enc(&planes.x, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(f32->base[0]), xd, xs, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return "cuTensorMapEncodeTiled(planes) failed";
        }
#define OTT_ROWS_LAUNCH(ACT)                                                                                                             \
    err = f32                 ? launch_variant<DT_S8_NHWC, ACT, kRowsQuantBuild>(stream, sm_count, planes, tmB, p, s, ep, out, status, to)  \
          : p.ctas_per_sm > 1 ? launch_variant<DT_S8_NHWC, ACT, kRowsBuild>(stream, sm_count, km, tmB, p, s, ep, out, status, to)       \
                              : launch_variant<DT_S8_NHWC, ACT, kRowsWideBuild>(stream, sm_count, km, tmB, p, s, ep, out, status, to)
        if (ep.int8_pos) OTT_ROWS_LAUNCH(ACT_POS);
        else if (ep.act_type == ACT_RELU) OTT_ROWS_LAUNCH(ACT_RELU);
        else if (ep.act_type == ACT_LRELU) OTT_ROWS_LAUNCH(ACT_LRELU);
        else if (ep.act_type == ACT_RELU6) OTT_ROWS_LAUNCH(ACT_RELU6);
        else OTT_ROWS_LAUNCH(ACT_NONE);
#undef OTT_ROWS_LAUNCH
    } else if (out_dtype == DT_S32_NHWC) {
        OTT_UMMA_LAUNCH(DT_S32_NHWC, ACT_NONE);
    } else if (out_dtype == DT_F32_NCHW) {
        OTT_UMMA_ACT(DT_F32_NCHW)
    } else if (ep.int8_pos && one_scale) {
        OTT_UMMA_LAUNCH(DT_S8_NHWC, ACT_POS | kOneScale);
    } else if (ep.int8_pos) {
        OTT_UMMA_LAUNCH(DT_S8_NHWC, ACT_POS);
    } else if (one_scale && ep.act_type == ACT_NONE) {
        OTT_UMMA_LAUNCH(DT_S8_NHWC, ACT_NONE | kOneScale);
    } else if (one_scale && ep.act_type == ACT_LRELU) {
        OTT_UMMA_LAUNCH(DT_S8_NHWC, ACT_LRELU | kOneScale);
    } else {
        OTT_UMMA_ACT(DT_S8_NHWC)
    }
#undef OTT_UMMA_ACT
#undef OTT_UMMA_LAUNCH
    if (err) return err;
    return cudaGetLastError() == cudaSuccess ? nullptr : "dense_umma_kernel launch failed";
}

}  // namespace ottk
