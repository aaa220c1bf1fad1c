// C5 masks with the dot products on the tensor cores (the variant that also returns the logits stays in kernels_yolact.cu).
//
// The answer is one bit per (detection, pixel): is the fp32 dot product of 32 terms above logit(thr)?  Formed exactly for every
// tile that a crop touches, in fp32 with the coefficients read as broadcasts from shared memory, a batch of 64 took 131 us against
// 43 us of traffic: the shared-memory pipe delivers one word per lane and cycle quarter, so two pixels per thread left the FMA
// units idle half the time, and masks left in two-byte stores.  Here:
//   - tcgen05 (bf16 operands split in two, the three products that matter, fp32 accumulators) gives every dot product within
//     2^-15 |p| |c| of its exact value, p and c being the pixel's and the detection's 32 values: each operand keeps 2^-18 of
//     itself in the two parts, lo * lo is left out (2^-18), and 96 additions in the accumulator lose less than 2^-16.3;
//     |sum p c| terms are bounded by |p| |c| (Cauchy).  A logit further than that (plus the rounding of the fp32 sigmoid) from
//     logit(thr) is decided; the others, about 2 in 10 000, are formed again in fp32 in the order of kernels_yolact.cu and
//     compared through the sigmoid, so the bytes are those of that kernel.
//   - A warp owns 32 pixels (TMEM lanes).  It forms the crop of every detection as a word of 32 bits (one detection per lane),
//     lists those that have any, and reads only their columns: a ballot gives the 32 comparisons of a column.  The masks leave
//     in aligned 16-byte pieces.  (All columns with the signs collected per pixel and transposed: 2170 instructions per 32
//     pixels and 100 detections, 141 us; issue was the bound.)
//   - A CTA of four warps walks neighbouring tiles of 128 pixels of one image; four CTAs per SM (128 TMEM columns each) overlap
//     one another's loads, products and stores.
//     (Two warps per 32 pixels, each with half of the detections: 115 us, what both have to do costs more than more warps bring.
//     TF32 operands, copied to shared memory unsplit, leave 1 in 100 logits open: 105 us.)
// B = 64, 138 x 138, 100 detections: 89 us (3.1 TB/s) against 129 for the exact kernel, each pass on other inputs; on the same ones
// 75 against 112, 8 x 276 x 276 42 against 57, one image 13 against 13.  What bounds it is issue, 1150 instructions per 32 pixels, with the 16 warps per SM that TMEM leaves room for.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>

#include "tcgen05.cuh"
#include "yolact.cuh"

namespace fb {

constexpr int kYtThreads = 128;
constexpr int kYtK = 32;
constexpr int kYtMaxDet = 256;
constexpr int kYtRow = 128;                    // bytes of one operand row: 32 hi, 32 lo bf16 values
constexpr int kYtTile = kYtThreads * kYtRow;   // 16 KB of pixels
constexpr int kYtBitsPitch = kYtMaxDet + 8;    // words per row of the bit table
constexpr uint32_t kYtWaitLimit = 2000000u;

// operand layout: no-swizzle K-major core matrices of 8 rows x 16 bytes, K-adjacent ones 128 bytes apart, 8-row groups 1024
__device__ __forceinline__ int yt_offset(int row, int chunk) { return (row >> 3) * 1024 + chunk * 128 + (row & 7) * 16; }

// Four consecutive values of a row as bf16 hi and lo parts: chunk = 16-byte chunk of the hi part, half = which 8 bytes of it.
__device__ __forceinline__ void yt_store_split(unsigned char* tile, int row, int chunk, int half, const float4 v) {
    const __nv_bfloat162 h0 = __floats2bfloat162_rn(v.x, v.y), h1 = __floats2bfloat162_rn(v.z, v.w);
    const uint32_t u0 = *reinterpret_cast<const uint32_t*>(&h0), u1 = *reinterpret_cast<const uint32_t*>(&h1);
    const __nv_bfloat162 l0 = __floats2bfloat162_rn(__fsub_rn(v.x, __uint_as_float(u0 << 16)), __fsub_rn(v.y, __uint_as_float(u0 & 0xffff0000u)));
    const __nv_bfloat162 l1 = __floats2bfloat162_rn(__fsub_rn(v.z, __uint_as_float(u1 << 16)), __fsub_rn(v.w, __uint_as_float(u1 & 0xffff0000u)));
    unsigned char* at = tile + yt_offset(row, chunk) + half * 8;
    *reinterpret_cast<uint2*>(at) = make_uint2(u0, u1);
    *reinterpret_cast<uint2*>(at + 4 * 128) = make_uint2(*reinterpret_cast<const uint32_t*>(&l0), *reinterpret_cast<const uint32_t*>(&l1));
}

// 32 rows of 32 floats, loaded by one warp: lane -> (row = (lane / 2) % 8 of eight, 32-byte piece lane / 16 of 64 bytes, half), so
// that a load takes whole sectors and the eight rows of a store fill all banks.  (base: the first row; rows: how many there are)
__device__ __forceinline__ void yt_load(const float* __restrict__ base, int rows, int lane, float4 (&v)[8]) {
    const int r = (lane >> 1) & 7;
    base += r * kYtK + (lane >> 4) * 8 + (lane & 1) * 4;
    if (rows >= 32) {
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = __ldg(reinterpret_cast<const float4*>(base + (q >> 1) * 8 * kYtK + (q & 1) * 16));
    } else {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            v[q] = (q >> 1) * 8 + r < rows ? __ldg(reinterpret_cast<const float4*>(base + (q >> 1) * 8 * kYtK + (q & 1) * 16))
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
// stores the split rows [row0, row0 + 32) of the tile; returns the sum of squares of row row0 + lane
__device__ __forceinline__ float yt_store(unsigned char* tile, int row0, int lane, const float4 (&v)[8]) {
    const int r = (lane >> 1) & 7;
    float sq[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        sq[g] = 0.0f;
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const float4 x = v[2 * g + p];
            yt_store_split(tile, row0 + g * 8 + r, p * 2 + (lane >> 4), lane & 1, x);
            sq[g] = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, fmaf(x.w, x.w, sq[g]))));
        }
        sq[g] += __shfl_xor_sync(kFullMask, sq[g], 1);
        sq[g] += __shfl_xor_sync(kFullMask, sq[g], 16);
    }
    float mine = 0.0f;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const float s = __shfl_sync(kFullMask, sq[g], (lane & 7) << 1);
        mine = (lane >> 3) == g ? s : mine;
    }
    return mine;
}

__device__ __forceinline__ void yt_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// eight TMEM columns, one 32-bit value each per lane
__device__ __forceinline__ void yt_columns(uint32_t taddr, uint2 list, float (&s)[8]) {
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        const uint32_t col = ((u < 4 ? list.x : list.y) >> (8 * (u & 3))) & 255u;
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=f"(s[u]) : "r"(taddr + col) : "memory");
    }
    // (the values are operands of the wait, so that nothing uses them before it)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+f"(s[0]), "+f"(s[1]), "+f"(s[2]), "+f"(s[3]), "+f"(s[4]), "+f"(s[5]), "+f"(s[6]), "+f"(s[7])::"memory");
}

// which of the 32 pixels from number p0 = y * width + x on lie in the crop (columns [b.x, b.y), rows [b.z, b.w))
__device__ __forceinline__ uint32_t yt_crop(const int4 b, int x, int y, int width) {
    uint32_t bits = 0u;
    for (int at = 0; at < 32; ++y) {
        const int n = min(width - x, 32 - at);
        const int lo = max(b.x - x, 0), len = max(min(b.y - x, n) - lo, 0);
        uint32_t run;
        asm("bmsk.clamp.b32 %0, %1, %2;" : "=r"(run) : "r"(at + lo), "r"(len));
        if (y >= b.z && y < b.w) bits |= run;
        at += n;
        x = 0;
    }
    return bits;
}

struct YtShared {
    uint64_t done;
    uint32_t tmem_base;
    float norm[kYtThreads / 32];
    int4 bounds[kYtMaxDet];
    uint32_t bits[8 * kYtBitsPitch];  // row r & 7: pixels [32 r, 32 r + 32) of the run, one word per detection
    __align__(8) uint8_t list[kYtThreads / 32][kYtMaxDet + 8];
};

// grid = (runs of tiles_per_cta tiles, images); dynamic shared memory: pixel tile, coefficient rows, YtShared
__global__ void __launch_bounds__(kYtThreads, 4)
yolact_masks_tc_kernel(const float* __restrict__ proto, const float* __restrict__ coef, const float* __restrict__ boxes, int height,
                       int width, int num_det, int n_mma, uint32_t tmem_cols, float thr, float mid, float slack, int tiles_per_cta,
                       uint8_t* __restrict__ masks) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* a_tile = smem_raw;
    unsigned char* b_tile = smem_raw + kYtTile;
    const int groups = (num_det + 31) >> 5;
    YtShared& sh = *reinterpret_cast<YtShared*>(b_tile + groups * 32 * kYtRow);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, img = blockIdx.y;
    const int hw = height * width;
    const float* pimg = proto + static_cast<int64_t>(img) * hw * kYtK;
    const float* cimg = coef + static_cast<int64_t>(img) * num_det * kYtK;

    const int tile0 = blockIdx.x * tiles_per_cta, tile1 = min(tile0 + tiles_per_cta, (hw + kYtThreads - 1) / kYtThreads);
    float4 v[8];
    {
        const int at = tile0 * kYtThreads + warp * 32;
        yt_load(pimg + static_cast<int64_t>(at) * kYtK, hw - at, lane, v);
    }
    if (t == 0) {
        mbar_init(&sh.done, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int d = t; d < num_det; d += kYtThreads) {
        const float4 bx = __ldg(reinterpret_cast<const float4*>(boxes) + static_cast<int64_t>(img) * num_det + d);
        int xs, xe, ys, ye;
        yolact_crop_range(bx.x, bx.z, width, xs, xe);
        yolact_crop_range(bx.y, bx.w, height, ys, ye);
        sh.bounds[d] = make_int4(xs, xe, ys, ye);
    }
    {
        float most = 0.0f;
        bool odd = false;  // a NaN does not survive a maximum
        for (int g = warp; g < groups; g += kYtThreads / 32) {
            float4 c[8];
            yt_load(cimg + g * 32 * kYtK, num_det - g * 32, lane, c);
            const float s = yt_store(b_tile, g * 32, lane, c);
            odd |= !(s < INFINITY);
            most = fmaxf(most, s);
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) most = fmaxf(most, __shfl_xor_sync(kFullMask, most, s));
        if (__any_sync(kFullMask, odd)) most = INFINITY;
        if (lane == 0) sh.norm[warp] = most;
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    const float cmax = fmaxf(fmaxf(sh.norm[0], sh.norm[1]), fmaxf(sh.norm[2], sh.norm[3]));
    // D = F32, A = B = BF16, both K-major, M = 128
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n_mma >> 3) << 17) | ((128u >> 4) << 24);
    bool usable = true;
    // a thread stores one 16-byte piece of every 16th detection: 16 planes on, the pieces lie on the same boundary
    uint8_t* plane0 = masks + (static_cast<int64_t>(img) * num_det + (t >> 3)) * hw;
    const int from = tile0 * kYtThreads, to = min(tile1 * kYtThreads, hw);

    for (int tile = tile0; tile < tile1; ++tile) {
        const float psq = yt_store(a_tile, warp * 32, lane, v);
        fence_proxy_async();
        tc_fence_before();
        __syncthreads();
        if (t == 0) {
            tc_fence_after();
            const uint32_t a = smem_u32(a_tile), b = smem_u32(b_tile);
            // k-steps of 16 values = two 16-byte chunks; hi parts at chunk 0, lo parts at chunk 4; the small products first
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const uint32_t ka = (i & 1) * 256 + (i < 2 ? 512 : 0), kb = (i & 1) * 256 + (i >= 2 && i < 4 ? 512 : 0);
                yt_mma(tmem, make_smem_desc(a + ka, 128, 1024), make_smem_desc(b + kb, 128, 1024), idesc, i > 0 ? 1u : 0u);
            }
            tc_commit(&sh.done);
        }
        const int p0 = tile * kYtThreads + warp * 32;
        const int y0 = p0 / width, x0 = p0 - y0 * width;
        if (tile + 1 < tile1) yt_load(pimg + static_cast<int64_t>(p0 + kYtThreads) * kYtK, hw - p0 - kYtThreads, lane, v);
        // the crops of this warp's 32 pixels, and a list of the detections that have any
        uint32_t* bits = sh.bits + ((4 * (tile - tile0) + warp) & 7) * kYtBitsPitch;
        int touched = 0;
        for (int g = 0; g < groups; ++g) {
            const int d = g * 32 + lane;
            const uint32_t crop = d < num_det ? yt_crop(sh.bounds[d], x0, y0, width) : 0u;
            bits[d] = crop;
            const uint32_t some = __ballot_sync(kFullMask, crop != 0u);
            if (crop != 0u) sh.list[warp][touched + __popc(some & ((1u << lane) - 1u))] = static_cast<uint8_t>(d);
            touched += __popc(some);
        }
        __syncwarp();
        if (touched > 0 && lane < 8) sh.list[warp][touched + lane] = sh.list[warp][touched - 1];  // the last batch repeats its last one
        __syncwarp();
        // (should the products not arrive, every logit counts as undecided)
        const bool arrived = usable && mbar_wait_bounded(&sh.done, static_cast<uint32_t>(tile - tile0) & 1u, kYtWaitLimit);
        usable = __all_sync(kFullMask, arrived);
        tc_fence_after();
        // 2^-15 and the rounding of this line; beyond 1e9 a part that underflows in one operand could matter in the other
        const float reach = usable && psq < 1e18f && cmax < 1e18f ? fmaf(sqrtf(psq * cmax), 3.06e-5f, slack) : INFINITY;
        const uint32_t taddr = tmem + (static_cast<uint32_t>(warp * 32) << 16);
#pragma unroll 1
        for (int i = 0; i < touched; i += 8) {
            const uint2 list = *reinterpret_cast<const uint2*>(&sh.list[warp][i]);
            float s[8];
            yt_columns(taddr, list, s);
            uint32_t mine = 0u;  // lane u: the pixels of detection u of the batch that lie above the threshold
            float over[8], least = INFINITY;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                over[u] = __fsub_rn(s[u], mid);
                const uint32_t above = __ballot_sync(kFullMask, over[u] > 0.0f);
                mine = lane == u ? above : mine;
                least = fminf(least, fabsf(over[u]));
            }
            const int d = sh.list[warp][i + (lane & 7)];
            uint32_t res = mine & bits[d];
            if (!__all_sync(kFullMask, least > reach)) {
                uint32_t open = 0u;
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t o = __ballot_sync(kFullMask, !(fabsf(over[u]) > reach));
                    open = lane == u ? o : open;
                }
                open &= bits[d];
                while (open) {
                    const int p = __ffs(open) - 1;
                    open &= open - 1;
                    const float* a = pimg + static_cast<int64_t>(p0 + p) * kYtK;
                    const float* c = cimg + d * kYtK;
                    float acc = 0.0f;
#pragma unroll 4
                    for (int k = 0; k < kYtK; k += 4) {
                        const float4 q = __ldg(reinterpret_cast<const float4*>(a + k)), w = __ldg(reinterpret_cast<const float4*>(c + k));
                        acc = fmaf(q.x, w.x, acc);
                        acc = fmaf(q.y, w.y, acc);
                        acc = fmaf(q.z, w.z, acc);
                        acc = fmaf(q.w, w.w, acc);
                    }
                    const uint32_t bit = 1u << p;
                    res = sigmoid_f32(acc) > thr ? res | bit : res & ~bit;
                }
            }
            __syncwarp();
            if (lane < 8) bits[d] = res;
        }
        tc_fence_before();
        __syncthreads();
        // Out in aligned pieces of 16 bytes, eight threads to a row: the piece that covers the boundary to the tile before takes
        // that tile's bits along; what lies outside this CTA's run is left to its neighbours.
        const int first = tile * kYtThreads, row0 = 4 * (tile - tile0);
        auto put = [&](uint8_t* plane, int d, int step, int piece) {
            const int at = piece * 16 - static_cast<int>(reinterpret_cast<uintptr_t>(plane + first) & 15);  // relative to the tile
            const int r = row0 + (at >> 5);  // (arithmetic shift: at = -1 .. -15 is the row before)
            const uint32_t* w0 = sh.bits + (r & 7) * kYtBitsPitch;
            const uint32_t* w1 = sh.bits + ((r + 1) & 7) * kYtBitsPitch;
            const int p = first + at;
            plane += p;
            if (p >= from && p + 16 <= to) {
#pragma unroll 2
                for (; d < num_det; d += step, plane += static_cast<int64_t>(step) * hw) {
                    const uint32_t w = __funnelshift_r(w0[d], w1[d], at);
                    uint4 o;
                    o.x = ((w & 15u) * 0x00204081u) & 0x01010101u;
                    o.y = (((w >> 4) & 15u) * 0x00204081u) & 0x01010101u;
                    o.z = (((w >> 8) & 15u) * 0x00204081u) & 0x01010101u;
                    o.w = (((w >> 12) & 15u) * 0x00204081u) & 0x01010101u;
                    *reinterpret_cast<uint4*>(plane) = o;
                }
            } else {  // planes and runs start at even addresses
                const int k0 = max(from - p, 0), k1 = min(16, to - p);
                if (k0 >= k1) return;
                for (; d < num_det; d += step, plane += static_cast<int64_t>(step) * hw) {
                    const uint32_t w = __funnelshift_r(w0[d], w1[d], at);
                    for (int k = k0; k < k1; k += 2)
                        *reinterpret_cast<uint16_t*>(plane + k) = static_cast<uint16_t>(((w >> k) & 1u) | (((w >> k) & 2u) << 7));
                }
            }
        };
        put(plane0, t >> 3, kYtThreads / 8, t & 7);
        if (tile + 1 == tile1)
            for (int d = t; d < num_det; d += kYtThreads) put(masks + (static_cast<int64_t>(img) * num_det + d) * hw, d, kYtMaxDet, 8);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols) : "memory");
}

int launch_yolact_masks_tc(const float* proto, const float* coef, const float* boxes, int batch, int height, int width, int num_det,
                           float thr, uint8_t* masks, cudaStream_t st) {
    const int groups = (num_det + 31) / 32, n_mma = (num_det + 15) / 16 * 16;
    uint32_t cols = 32;
    while (cols < static_cast<uint32_t>(groups * 32)) cols *= 2;
    const int per_sm = std::min(4, static_cast<int>(512 / cols));
    const size_t smem = kYtTile + static_cast<size_t>(groups) * 32 * kYtRow + sizeof(YtShared);
    FB_TRY(check_cuda(cudaFuncSetAttribute(yolact_masks_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           kYtTile + kYtMaxDet * kYtRow + static_cast<int>(sizeof(YtShared))), "yolact_masks_tc attr"));
    // one wave of CTAs, each with as many neighbouring tiles of an image as that takes
    const int tiles = static_cast<int>((static_cast<int64_t>(height) * width + kYtThreads - 1) / kYtThreads);
    const int64_t slots = static_cast<int64_t>(kNumSMs) * per_sm;
    const int per_image = static_cast<int>(std::max<int64_t>(1, slots / batch));
    const int run = (tiles + per_image - 1) / per_image;
    const dim3 grid(static_cast<unsigned>((tiles + run - 1) / run), static_cast<unsigned>(batch));
    const double mid = std::log(static_cast<double>(thr) / (1.0 - static_cast<double>(thr)));
    // the fp32 sigmoid is within 4.2e-7 of itself of the exact one: a logit 4.2e-7 / (1 - thr) from the threshold is on its
    // side.  Ten times that.
    const double slack = 4.0e-6 / (static_cast<double>(thr) * (1.0 - static_cast<double>(thr)));
    yolact_masks_tc_kernel<<<grid, kYtThreads, smem, st>>>(proto, coef, boxes, height, width, num_det, n_mma, cols, thr,
                                                           static_cast<float>(mid), static_cast<float>(slack), run, masks);
    count_launch();
    return check_launch("yolact_masks_tc_kernel");
}

}  // namespace fb
