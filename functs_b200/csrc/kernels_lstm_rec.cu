// C4, the recurrence: one thread-block cluster of 16 CTAs owns a few batch rows and runs all time steps on its own.
//
// The rows of a batch are independent, so nothing but the 16 CTAs that share a row's hidden state has to meet between steps.  h goes
// into the others' shared memory by st.async, 16 bytes and their count on the receiver's mbarrier in one store: 0.7 us per step
// at one row of H = 256 (plain remote stores, a fence and a cluster barrier 1.2; one bulk copy per receiver 1.6).  Every cluster holds all of w_hh: a CTA owns H / 16 hidden units,
// four gate columns each, 64 KB (H = 256) or 256 KB (H = 512) of weights, in registers as far as they go (32 or 64 per thread),
// the rest in shared memory.
// What bounds it at 64 rows: seven clusters fit the chip, ten rows each; of 4.2 us per step (5.6 before the two halves took turns) 2.6
// are fp32 multiply-adds at 128 per cycle and SM, the rest is what their operands' loads and the gates take of the same issue slots;
// at one row the latency of a step: multiply 300 cycles, sum 240, gates 290, send and arrive 450.
//
// Thread layout: a thread multiplies two gate columns of one unit with KT consecutive k of every row, two k per packed instruction
// (fma.rn.f32x2: one issue slot for two multiply-adds); a warp is 8 units x 2 gate pairs x 2 k-slices, the two slices are
// summed by a shuffle that leaves one gate per lane, the warps' sums meet in shared memory, and one thread per (row, unit)
// applies the gates, assigns hs[t] / cs[t] and sends h into the sixteen CTAs' next buffer.  (Four gate columns and half the k
// per thread needs two passes over the rows, and the weights in shared memory are then read twice: 6.5 us per step at ten
// rows of H = 512.  A register spill here goes to L2, shared memory being full: 14 us.)
#include "common.cuh"

namespace fb {

constexpr int kRecCluster = 16;
constexpr int kRecThreads = 512;
constexpr int kRecUnitsPerWarp = 8;
constexpr int kRecSlices = 2;  // k-slices inside a warp
constexpr int kRecAhead = 2;   // steps that the projection's values are fetched ahead
constexpr uint32_t kRecWaitLimit = 250000u;  // about a second: a poll that fails takes 7800 cycles
// Development switch (functs_b200_debug_set "lstm_drop_exchange"): in this thread's calls no CTA sends h, so that every wait runs out.
static thread_local int t_rec_drop = 0;
void lstm_set_drop_exchange(int on) { t_rec_drop = on ? 1 : 0; }
// Steps and rows up to which a cluster forms its own projection: 0.18 us per row at an input of 256 instead of a kernel in front of it, whose
// time grows with the depth faster than the cluster's does.  Two launches / one, us between two calls, inputs of 64, 256 and 512: 4 steps of
// one row 12.4 / 8.4, 17.1 / 10.4, 22.7 / 10.4; 25 of one 27.6 / 26.8, 33.0 / 28.8, 39.1 / 30.9; 56 of one 50.0 / 51.4, 55.5 / 55.5,
// 62.2 / 61.7; 56 of seven 53.5 / 51.4, 59.6 / 55.5, 69.8 / 61.9; 32 of fourteen 41.1 / 39.1, 47.3 / 43.2, 56.9 / 53.5.  Beyond (256):
// 64 of one 72 / 73 a call, 64 of two 88 / 94.  (Inputs of 16 and 64 lose up to 4 % from 40 steps of one row on.)  H = 512 has no such form:
// half of its weights lie in shared memory, and the partial sums of rec_project would take 128 KB beside them.
constexpr int kOneLaunchSteps = 56, kOneLaunchRows = 64;

template <int H, int R>
struct RecLayout {
    static constexpr int U = H / kRecCluster;                       // units per CTA
    static constexpr int WG = U / kRecUnitsPerWarp;                 // warps across the units
    static constexpr int KQ = kRecThreads / 32 / WG;                // k-ranges across the warps
    static constexpr int KT = H / KQ / kRecSlices;                  // k per thread
    static constexpr int BP = R * U + 4;                            // a CTA's part of h, [R][U], and four floats (banks)
    static constexpr int Quads = KT / 4;
    static constexpr int RegQuads = Quads < 8 ? Quads : 8;          // k-quads whose weights live in registers
    static constexpr int SmemQuads = Quads - RegQuads;
    static constexpr size_t h_floats = 2ull * kRecCluster * BP;
    static constexpr size_t part_floats = static_cast<size_t>(KQ) * R * 4 * U;
    static constexpr size_t w_bytes = static_cast<size_t>(SmemQuads) * 2 * kRecThreads * 16;
    static constexpr int Items = R * U;                             // (row, unit) pairs of the CTA
    static constexpr int GateWarps = (Items + 31) / 32;
    static constexpr int Sends = kRecCluster * (Items / 4) / (GateWarps * 32);  // CTAs that a gate thread sends a quad of units to
    static constexpr size_t pre_floats = (kRecAhead + 1ull) * Items * 4;        // [step][R][4][U]
    static constexpr size_t bytes = w_bytes + (h_floats + part_floats + pre_floats) * 4 + 32;
    static_assert(KT % U == 0, "a k-slice is whole parts of h");
    static_assert(Items % 16 == 0 && Items / 4 * kRecCluster == Sends * GateWarps * 32, "every gate thread sends");
};

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float sum2(unsigned long long v) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
    return __fadd_rn(lo, hi);
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Address of this CTA's shared-memory word in the CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_remote(uint32_t local_addr, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local_addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void store_async4(uint32_t remote, float a, float b, float c, float d, uint32_t remote_bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(remote), "f"(a),
                 "f"(b), "f"(c), "f"(d), "r"(remote_bar)
                 : "memory");
}
// Wait for what other CTAs of the cluster store; false when the limit runs out.
//
// What follows then, in both kernels.  The warp multiplies no more and goes through the named barriers of the steps that are left, in
// step with the gate warps: barrier.arrive would let it run ahead, and a barrier that a warp meets twice in one phase loses count,
// so that the gate warps wait for ever.  (The barrier of the step before is over by then: the other warps of its CTA have seen the same h
// a second ago.)  The outputs then mean nothing, which the status word says.  A CTA whose gate warps, or whose thread that sets the
// mbarriers for the next round, gave up sends no whole h any more: a gate warp that gave up sends none, and in the second
// kernel, whose gate warps never wait, they see `late` behind the barrier.  So no mbarrier receives more than it expects, and the
// waits of the other CTAs run out in their turn, once per warp.
__device__ __forceinline__ bool wait_cluster(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kRecWaitLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// Phase of a buffer's mbarrier that step t waits for: steps 1, 3, 5, ... use buffer 1, steps 2, 4, ... buffer 0.
__device__ __forceinline__ uint32_t step_parity(int t) { return static_cast<uint32_t>((t - 1) >> 1) & 1u; }

// (not the .aligned forms: the lanes of a warp come here from different sides of a branch)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

// The input projection of a cluster's few rows, by the cluster itself (PQ > 0: ceil(K / 128) for H = 256): every CTA forms the columns
// of its own units for all steps, so that nothing is launched and nothing goes through global memory in front of the first step.
struct RecInput {
    const float *x, *w_ih, *b_ih, *b_hh;
    int K;
};
template <int H, int R, int PQ>
struct ProjLayout {
    static constexpr int U = H / kRecCluster;
    static constexpr int Slices = kRecThreads / U;                  // k-slices: a thread takes four columns of a unit and 4 * PQ k
    static constexpr int Kp = Slices * 4 * PQ;                      // the depth, zeros behind K
    static constexpr int Rows = 16;                                 // at a time
    static constexpr size_t x_floats = static_cast<size_t>(Rows) * Kp;
    static constexpr size_t part_floats = static_cast<size_t>(kRecThreads / 32) * Rows * U * 4;
    static size_t bytes(int steps) {  // in place of RecLayout's ring
        return RecLayout<H, R>::bytes + (static_cast<size_t>(steps) * R * U * 4 + x_floats + part_floats - RecLayout<H, R>::pre_floats) * 4;
    }
    static_assert((U == 16 && Rows % 2 == 0) || PQ == 0, "two slices in a warp");
};
// pre_all: [T][R][4][U]; x_s: [Rows][Kp]; part: [warps][Rows][U][4].  fp32 sums of 4 * PQ products per thread, 2 * warps of them added.
template <int H, int R, int PQ>
__device__ __forceinline__ void rec_project(const RecInput& in, int T, int B, int b0, int j0, float* pre_all, float* x_s, float* part) {
    using P = ProjLayout<H, R, PQ>;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int unit = tid % P::U, k0 = tid / P::U * (4 * PQ);
    unsigned long long w[PQ][4][2];
#pragma unroll
    for (int q = 0; q < PQ; ++q)
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int k = k0 + 4 * q + i;
                v[i] = k < in.K ? __ldg(in.w_ih + (static_cast<int64_t>(g) * in.K + k) * H + j0 + unit) : 0.0f;
            }
            w[q][g][0] = pack2(v[0], v[1]);
            w[q][g][1] = pack2(v[2], v[3]);
        }
    const int rows = T * R;
    for (int r0 = 0; r0 < rows; r0 += P::Rows) {
        const int most = min(P::Rows, rows - r0);
        for (int e = tid; e < most * P::Kp; e += kRecThreads) {
            const int i = e / P::Kp, k = e - i * P::Kp, t = (r0 + i) / R, row = b0 + (r0 + i) % R;
            x_s[e] = k < in.K && row < B ? __ldg(in.x + (static_cast<int64_t>(t) * B + row) * in.K + k) : 0.0f;
        }
        __syncthreads();
        // two rows at a time: the lower half of a warp ends with the sums of the first one, the upper half with those of the second
        // (an odd last row takes whatever lies behind it along)
        const bool up = lane >= 16;
        for (int i = 0; i < most; i += 2) {
            unsigned long long acc[2][4] = {};
#pragma unroll
            for (int q = 0; q < PQ; ++q) {
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const ulonglong2 xv = *reinterpret_cast<const ulonglong2*>(x_s + (i + r) * P::Kp + k0 + 4 * q);
#pragma unroll
                    for (int g = 0; g < 4; ++g) acc[r][g] = fma2(xv.y, w[q][g][1], fma2(xv.x, w[q][g][0], acc[r][g]));
                }
            }
            float s[4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float s0 = sum2(acc[0][g]), s1 = sum2(acc[1][g]);
                s[g] = __fadd_rn(up ? s1 : s0, __shfl_xor_sync(kFullMask, up ? s0 : s1, 16));
            }
            reinterpret_cast<float4*>(part)[(warp * P::Rows + i + (up ? 1 : 0)) * P::U + unit] = make_float4(s[0], s[1], s[2], s[3]);
        }
        __syncthreads();
        for (int e = tid; e < most * P::U; e += kRecThreads) {
            const int i = e / P::U, u = e - i * P::U;
            float4 s = reinterpret_cast<const float4*>(part)[e];
#pragma unroll
            for (int v = 1; v < kRecThreads / 32; ++v) {
                const float4 m = reinterpret_cast<const float4*>(part)[v * P::Rows * P::U + e];
                s.x = __fadd_rn(s.x, m.x);
                s.y = __fadd_rn(s.y, m.y);
                s.z = __fadd_rn(s.z, m.z);
                s.w = __fadd_rn(s.w, m.w);
            }
            const float sums[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
            for (int g = 0; g < 4; ++g)
                pre_all[((r0 + i) * 4 + g) * P::U + u] =
                    __fadd_rn(sums[g], __fadd_rn(__ldg(in.b_ih + g * H + j0 + u), __ldg(in.b_hh + g * H + j0 + u)));
        }
        // (the next rows' barrier stands between these reads of part and its next stores)
    }
    __syncthreads();
}

// R rows per cluster, multiplied in one pass.  PQ: see ProjLayout; 0: the projection is in `pre`.
template <int H, int R, int PQ>
__global__ void __launch_bounds__(kRecThreads, 1)
lstm_recurrent_kernel(const float* __restrict__ pre, const float* __restrict__ w_hh, int T, int B, float* __restrict__ hs,
                      float* __restrict__ cs, int32_t* status, int drop_exchange, const RecInput in) {
    using Y = RecLayout<H, R>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ulonglong2* w_s = reinterpret_cast<ulonglong2*>(smem_raw);                  // [SmemQuads][2][kRecThreads]
    float* h_s = reinterpret_cast<float*>(smem_raw + Y::w_bytes);               // [2][16][BP]
    float* part = h_s + Y::h_floats;                                            // [KQ][R][U][4]
    uint64_t* full = reinterpret_cast<uint64_t*>(part + Y::part_floats);        // [buffer]
    int* late = reinterpret_cast<int*>(full + 2);                               // a wait ran out
    float* pre_s = reinterpret_cast<float*>(full + 4);                          // [PQ > 0 ? step : step % 3][R][4][U]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = static_cast<int>(cluster_rank());
    const int b0 = static_cast<int>(blockIdx.x / kRecCluster) * R;
    const int unit = (warp % Y::WG) * kRecUnitsPerWarp + (lane & 7);            // of this CTA
    const int gates = (lane >> 2) & 2;                                          // first of this thread's two gates
    const int kq = warp / Y::WG, slice = kq * kRecSlices + (lane >> 4);         // k = slice * KT ...
    const int j0 = rank * Y::U;
    constexpr uint32_t kPhaseBytes = R * H * 4;                                 // all of h
    if (tid == 0) {
        *late = 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            mbar_init(full + i, 1);
            mbar_arrive_expect_tx(full + i, kPhaseBytes);
        }
        fence_barrier_init();
    }

    // resident weights: gate c, k -> w_hh[c][k][j0 + unit]
    unsigned long long w_r[Y::RegQuads][2][2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const float* src = w_hh + (static_cast<int64_t>(gates + c) * H + slice * Y::KT) * H + j0 + unit;
#pragma unroll
        for (int q = 0; q < Y::Quads; ++q) {
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = __ldg(src + static_cast<int64_t>(4 * q + i) * H);
            if (q < Y::RegQuads) {
                w_r[q < Y::RegQuads ? q : 0][c][0] = pack2(v[0], v[1]);
                w_r[q < Y::RegQuads ? q : 0][c][1] = pack2(v[2], v[3]);
            } else {
                w_s[((q - Y::RegQuads) * 2 + c) * kRecThreads + tid] = make_ulonglong2(pack2(v[0], v[1]), pack2(v[2], v[3]));
            }
        }
    }
    if constexpr (PQ > 0) {
        float* x_s = pre_s + static_cast<size_t>(T) * R * Y::U * 4;
        rec_project<H, R, PQ>(in, T, B, b0, j0, pre_s, x_s, x_s + ProjLayout<H, R, PQ>::x_floats);
    }
    // the first warps: one thread per (row, unit) of the CTA applies the gates, keeps the cell state and writes the outputs
    const bool gating = warp < Y::GateWarps, item = tid < Y::Items;
    const int i = item ? tid : 0, iu = i % Y::U, row = b0 + i / Y::U;
    float c_state = 0.0f;
    // 16 bytes a thread: gate (tid % U) / (U / 4), four units
    auto fetch = [&](int t) {
        if (PQ > 0) return;
        if (item && t < T) {
            const int g = iu / (Y::U / 4), u = iu % (Y::U / 4) * 4;
            const float* p = pre + (static_cast<int64_t>(t) * B + (row < B ? row : 0)) * (4 * H) + g * H + j0 + u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(pre_s + ((t % (kRecAhead + 1)) * Y::Items + i) * 4)), "l"(p)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // what this thread sends: a quad of units to Sends CTAs
    const int per_quad = kRecCluster / Y::Sends, quad = lane / per_quad;
    uint32_t dst[Y::Sends];
#pragma unroll
    for (int k = 0; k < Y::Sends; ++k)
        dst[k] = map_remote(smem_u32(smem_raw), static_cast<uint32_t>(lane % per_quad * Y::Sends + k));
    const uint32_t h_off = smem_u32(h_s + rank * Y::BP + warp * 32 + quad * 4) - smem_u32(smem_raw);
    const uint32_t bar_off = smem_u32(full) - smem_u32(smem_raw);
    if (gating) {
        if (PQ == 0) pdl_wait();  // the projection; the weights are not its output
#pragma unroll
        for (int t = 0; t < kRecAhead; ++t) fetch(t);
    }
    cluster_arrive();  // every CTA of the cluster runs, its barriers set, before anybody stores into another one
    cluster_wait();
    for (int t = 0; t < T; ++t) {
        if (t > 0) {
            if (!__all_sync(kFullMask, wait_cluster(smem_u32(full + (t & 1)), step_parity(t)))) {
                *late = 1;  // (see wait_cluster)
                if (lane == 0 && status != nullptr) atomicOr(status, FB_STATUS_WAIT_TIMEOUT);
                __syncwarp();
                for (; t < T; ++t) asm volatile("barrier.sync 1, %0;" ::"n"(kRecThreads) : "memory");
                break;
            }
            if (tid == 0 && t + 2 < T) mbar_arrive_expect_tx(full + (t & 1), kPhaseBytes);
            const float* h_t = h_s + ((t & 1) * kRecCluster + slice * (Y::KT / Y::U)) * Y::BP;
            unsigned long long acc[2][R];
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int r = 0; r < R; ++r) acc[c][r] = 0ull;
            auto quad = [&](const float* hq, const ulonglong2& w0, const ulonglong2& w1) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const ulonglong2 hv = *reinterpret_cast<const ulonglong2*>(hq + r * Y::U);
                    acc[0][r] = fma2(hv.x, w0.x, acc[0][r]);
                    acc[1][r] = fma2(hv.x, w1.x, acc[1][r]);
                    acc[0][r] = fma2(hv.y, w0.y, acc[0][r]);
                    acc[1][r] = fma2(hv.y, w1.y, acc[1][r]);
                }
            };
#pragma unroll
            for (int q = 0; q < Y::RegQuads; ++q)
                quad(h_t + (4 * q / Y::U) * Y::BP + 4 * q % Y::U, make_ulonglong2(w_r[q][0][0], w_r[q][0][1]),
                     make_ulonglong2(w_r[q][1][0], w_r[q][1][1]));
#pragma unroll 2
            for (int q = 0; q < Y::SmemQuads; ++q) {
                const int k = 4 * (Y::RegQuads + q);
                quad(h_t + (k / Y::U) * Y::BP + k % Y::U, w_s[(q * 2) * kRecThreads + tid], w_s[(q * 2 + 1) * kRecThreads + tid]);
            }
            // sum of the warp's two k-slices: afterwards a lane of the upper half holds its second gate, of the lower its first
            const bool up = (lane & 16) != 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float v0 = sum2(acc[0][r]), v1 = sum2(acc[1][r]);
                const float b = __fadd_rn(up ? v1 : v0, __shfl_xor_sync(kFullMask, up ? v0 : v1, 16));
                part[((kq * R + r) * Y::U + unit) * 4 + gates + (lane >> 4)] = b;
            }
        }
        // the partial sums of all warps, the fetched values of the gate warps; the other warps go on to the next step
        if (!gating) {
            __syncwarp();
            asm volatile("barrier.arrive 1, %0;" ::"n"(kRecThreads) : "memory");
            continue;
        }
        float gate[4];
        const float* pre_t = pre_s + (PQ > 0 ? t : t % (kRecAhead + 1)) * (Y::Items * 4) + i / Y::U * (4 * Y::U) + iu;
        if (PQ > 0) {
#pragma unroll
            for (int g = 0; g < 4; ++g) gate[g] = pre_t[g * Y::U];
        } else {
            asm volatile("cp.async.wait_group %0;" ::"n"(kRecAhead - 1) : "memory");
        }
        __syncwarp();
        asm volatile("barrier.sync 1, %0;" ::"n"(kRecThreads) : "memory");
        if (PQ == 0) {
#pragma unroll
            for (int g = 0; g < 4; ++g) gate[g] = pre_t[g * Y::U];
        }
        if (t > 0) {
            const float4* p = reinterpret_cast<const float4*>(part) + i;
            float4 s = p[0];
#pragma unroll
            for (int k = 1; k < Y::KQ; ++k) {
                const float4 v = p[k * Y::Items];
                s.x = __fadd_rn(s.x, v.x);
                s.y = __fadd_rn(s.y, v.y);
                s.z = __fadd_rn(s.z, v.z);
                s.w = __fadd_rn(s.w, v.w);
            }
            gate[0] = __fadd_rn(gate[0], s.x);
            gate[1] = __fadd_rn(gate[1], s.y);
            gate[2] = __fadd_rn(gate[2], s.z);
            gate[3] = __fadd_rn(gate[3], s.w);
        }
        float sg[3] = {gate[0], gate[1], gate[3]};
        sigmoid_f32_n(sg);
        const float ig = sg[0], fg = sg[1], og = sg[2], gg = tanhf(gate[2]);
        c_state = __fadd_rn(__fmul_rn(fg, c_state), __fmul_rn(ig, gg));
        const float hval = __fmul_rn(og, tanhf(c_state));
        if (t + 1 < T) {
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = __shfl_sync(kFullMask, hval, quad * 4 + k);
            const uint32_t to = h_off + static_cast<uint32_t>(((t + 1) & 1) * (kRecCluster * Y::BP)) * 4;
            const uint32_t bar = bar_off + static_cast<uint32_t>((t + 1) & 1) * 8;
            if (!drop_exchange) {
#pragma unroll
                for (int k = 0; k < Y::Sends; ++k) store_async4(dst[k] + to, v[0], v[1], v[2], v[3], dst[k] + bar);
            }
        }
        if (item && row < B) {
            const int64_t o = (static_cast<int64_t>(t) * B + row) * H + j0 + iu;
            hs[o] = hval;
            cs[o] = c_state;
        }
        fetch(t + kRecAhead);  // (into the place of step t - 1, which all gate threads have read)
    }
    if (PQ == 0) asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_arrive();  // nobody leaves while another CTA may still store into its shared memory
    cluster_wait();
    if (*late) {       // (stores of h that nobody waited for may be under way; they arrive within microseconds)
        const unsigned long long t0 = clock64();
        while (clock64() - t0 < 400000ull) {
        }
    }
}

// ---- many rows per cluster ----
// With more than a few rows the loads of h bound the kernel above: a 16-byte shared load fills 512 bytes of registers whatever
// its lanes share, four cycles, and feeds two gate columns only.  Here 256 threads of most of the registers take eight columns
// each, the four gates of two neighbouring units, packed by unit (a weight pair is adjacent in memory; h is the same in both
// halves), so that a loaded word feeds eight multiply-adds.
//
// The rows of a cluster are two halves that take turns: while eight warps multiply one half, eight others reduce, apply the gates
// and exchange the h of the other, so that the chain of a step (reduction, gates, exchange) lies behind multiplications instead of
// after them.  The exchange is st.async: 16 bytes and their count on the receiver's mbarrier in one store, no fence, no cluster
// barrier.  Nothing else orders the CTAs: a CTA can send h[t + 2] into a buffer only after it received all of h[t + 1], which every
// CTA sends after its own multiplications of h[t] have ended; the partial sums have one buffer per half for the same reason.
constexpr int kPairFma = 256, kPairGate = 256, kPairThreads = kPairFma + kPairGate;
constexpr int kPairFmaRegs = 200, kPairGateRegs = 56;               // of 128 per thread at launch
static_assert((kPairFmaRegs + kPairGateRegs) * 256 <= kPairThreads * 128, "registers of the launch");

template <int H, int RH>                                            // RH: rows of a half
struct PairLayout {
    static constexpr int U = H / kRecCluster;                       // units per CTA
    static constexpr int WG = U / 16;                               // warps across the units: 8 pairs per warp
    static constexpr int KQ = kPairFma / 32 / WG;                   // k-ranges across the warps
    static constexpr int KT = H / KQ / 4;                           // k per thread: four slices inside a warp
    static constexpr int BP = RH * U + 4;                           // a CTA's part of a half of h, [RH][U], and four floats (banks)
    static constexpr int RegK = KT <= 14 ? KT : 14;                 // k whose weights live in registers
    static constexpr int SmemK = KT - RegK;
    static constexpr int Items = RH * U;                            // (row, unit) pairs of a half
    static constexpr int GateWarps = (Items + 31) / 32;
    static constexpr size_t h_floats = 4ull * kRecCluster * BP;     // [buffer][half]
    static constexpr size_t part_floats = 2ull * KQ * RH * 4 * U;   // [half]
    static constexpr size_t w_bytes = static_cast<size_t>(SmemK) * 2 * kPairFma * 16;
    static constexpr size_t pre_floats = (kRecAhead + 1ull) * 2 * RH * 4 * U;  // [step][half][RH][4][U]
    static constexpr size_t bytes = w_bytes + (h_floats + part_floats + pre_floats) * 4 + 64;
    static_assert(U % KT == 0 && RegK % 2 == 0 && SmemK % 2 == 0, "a k-slice lies inside one part of h");
    static_assert(GateWarps * 32 <= kPairGate, "one thread per item");
};

template <int H, int RH>
__global__ void __launch_bounds__(kPairThreads, 1)
lstm_recurrent_pair_kernel(const float* __restrict__ pre, const float* __restrict__ w_hh, int T, int B, float* __restrict__ hs,
                           float* __restrict__ cs, int32_t* status, int drop_exchange) {
    using Y = PairLayout<H, RH>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ulonglong2* w_s = reinterpret_cast<ulonglong2*>(smem_raw);                  // [SmemK][2][kPairFma]
    float* h_s = reinterpret_cast<float*>(smem_raw + Y::w_bytes);               // [buffer][half][16][BP]
    float* part = h_s + Y::h_floats;                                            // [half][KQ][RH][U][4]
    float* pre_s = part + Y::part_floats;                                       // [step % 3][half][RH][4][U]
    uint64_t* full = reinterpret_cast<uint64_t*>(pre_s + Y::pre_floats);        // [half][buffer]
    volatile int* late = reinterpret_cast<int*>(full + 4);                      // a wait ran out
    const int tid = threadIdx.x, lane = tid & 31;
    const int rank = static_cast<int>(cluster_rank());
    const int b0 = static_cast<int>(blockIdx.x / kRecCluster) * (2 * RH);
    const int j0 = rank * Y::U;
    constexpr uint32_t kPhaseBytes = RH * H * 4;                                // one half of h

    if (tid == 0) {
        *late = drop_exchange;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            mbar_init(full + i, 1);
            mbar_arrive_expect_tx(full + i, kPhaseBytes);
        }
        fence_barrier_init();
    }
    if (tid < kPairFma) {
        // ---- multiplications ----
        __syncwarp();
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPairFmaRegs));
        const int warp = tid >> 5;
        const int unit = (warp % Y::WG) * 16 + 2 * (lane & 7);                  // first of this thread's two units
        const int kq = warp / Y::WG, slice = kq * 4 + (lane >> 3);              // k = slice * KT ...
        unsigned long long w_r[Y::RegK][4];
#pragma unroll
        for (int k = 0; k < Y::KT; ++k) {
            unsigned long long v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c)
                v[c] = __ldg(reinterpret_cast<const unsigned long long*>(w_hh + (static_cast<int64_t>(c) * H + slice * Y::KT + k) * H + j0 + unit));
            if (k < Y::RegK) {
#pragma unroll
                for (int c = 0; c < 4; ++c) w_r[k < Y::RegK ? k : 0][c] = v[c];
            } else {
                w_s[((k - Y::RegK) * 2) * kPairFma + tid] = make_ulonglong2(v[0], v[1]);
                w_s[((k - Y::RegK) * 2 + 1) * kPairFma + tid] = make_ulonglong2(v[2], v[3]);
            }
        }
        cluster_arrive();  // every CTA of the cluster runs, its barriers set, before anybody stores into another one
        cluster_wait();
        auto give_up = [&](int u) {  // (see wait_cluster)
            *late = 1;
            if (lane == 0 && status != nullptr) atomicOr(status, FB_STATUS_WAIT_TIMEOUT);
            __syncwarp();
            for (; u < 2 * T; ++u) asm volatile("barrier.sync %0, %1;" ::"r"(1 + (u & 1)), "n"(kPairFma + Y::GateWarps * 32) : "memory");
        };
        // Whether all lanes' waits ended well is asked after the multiplications, where it replaces a __syncwarp; at H = 512 there is no
        // register to keep the answer (64 steps of 64 rows, us: asked first 140.3 at H = 256, 338.6 at 512; later 139.4, 340.3).
        constexpr bool kVoteFirst = H == 512;
        // slice s lies in the part of CTA s * KT / U
        const float* h_mine = h_s + (slice * Y::KT / Y::U) * Y::BP + slice * Y::KT % Y::U;
#pragma unroll 1
        for (int u = 2; u < 2 * T; ++u) {                                       // (step, half)
            const int t = u >> 1, half = u & 1;
            uint64_t* bar = full + half * 2 + (t & 1);
            const bool ok = wait_cluster(smem_u32(bar), step_parity(t));
            if (kVoteFirst && !__all_sync(kFullMask, ok)) {
                give_up(u);
                break;
            }
            if (tid == 0 && ok && t + 2 < T) mbar_arrive_expect_tx(bar, kPhaseBytes);
            const float* h_t = h_mine + ((t & 1) * 2 + half) * (kRecCluster * Y::BP);
            unsigned long long acc[4][RH];
#pragma unroll
            for (int c = 0; c < 4; ++c)
#pragma unroll
                for (int r = 0; r < RH; ++r) acc[c][r] = 0ull;
            auto pair = [&](const float* hk, const unsigned long long (&w0)[4], const unsigned long long (&w1)[4]) {
#pragma unroll
                for (int r = 0; r < RH; ++r) {
                    const float2 hv = *reinterpret_cast<const float2*>(hk + r * Y::U);
                    const unsigned long long x = pack2(hv.x, hv.x), y = pack2(hv.y, hv.y);
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c][r] = fma2(x, w0[c], acc[c][r]);
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c][r] = fma2(y, w1[c], acc[c][r]);
                }
            };
#pragma unroll
            for (int k = 0; k < Y::RegK; k += 2) pair(h_t + k, w_r[k], w_r[k + 1 < Y::RegK ? k + 1 : k]);
#pragma unroll
            for (int k = 0; k < Y::SmemK; k += 2) {
                const ulonglong2 a0 = w_s[(2 * k) * kPairFma + tid], a1 = w_s[(2 * k + 1) * kPairFma + tid];
                const ulonglong2 b0_ = w_s[(2 * k + 2) * kPairFma + tid], b1_ = w_s[(2 * k + 3) * kPairFma + tid];
                const unsigned long long w0[4] = {a0.x, a0.y, a1.x, a1.y}, w1[4] = {b0_.x, b0_.y, b1_.x, b1_.y};
                pair(h_t + Y::RegK + k, w0, w1);
            }
            // sum over the warp's four k-slices: after the two exchanges a lane holds two gates of one of its units
            const bool up = (lane & 16) != 0, odd = (lane & 8) != 0;
#pragma unroll
            for (int r = 0; r < RH; ++r) {
                float a[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    float u0, u1;
                    asm("mov.b64 {%0, %1}, %2;" : "=f"(u0), "=f"(u1) : "l"(acc[c][r]));
                    a[c] = __fadd_rn(up ? u1 : u0, __shfl_xor_sync(kFullMask, up ? u0 : u1, 16));
                }
                const float s0 = __fadd_rn(odd ? a[2] : a[0], __shfl_xor_sync(kFullMask, odd ? a[0] : a[2], 8));
                const float s1 = __fadd_rn(odd ? a[3] : a[1], __shfl_xor_sync(kFullMask, odd ? a[1] : a[3], 8));
                *reinterpret_cast<float2*>(part + (((half * Y::KQ + kq) * RH + r) * Y::U + unit + (lane >> 4)) * 4 + (odd ? 2 : 0)) =
                    make_float2(s0, s1);
            }
            if (kVoteFirst) {
                __syncwarp();
            } else if (!__all_sync(kFullMask, ok)) {
                give_up(u);
                break;
            }
            asm volatile("barrier.arrive %0, %1;" ::"r"(1 + half), "n"(kPairFma + Y::GateWarps * 32) : "memory");
        }
    } else {
        // ---- gates and exchange: one thread per (row, unit) of a half ----
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPairGateRegs));
        cluster_arrive();
        // The first half's items are on the first warps, the second half's on the last ones: no scheduler has the odd warp of both.
        const int gw = (tid - kPairFma) >> 5;
        if (gw < Y::GateWarps || gw >= kPairGate / 32 - Y::GateWarps) {
            int item[2];                                                        // (row, unit) of each half, or -1
            item[0] = tid - kPairFma;
            item[1] = item[0] - (kPairGate - Y::GateWarps * 32);
            const bool mine[2] = {gw < Y::GateWarps, item[1] >= 0};             // the warp has items of this half
#pragma unroll
            for (int half = 0; half < 2; ++half) item[half] = item[half] < Y::Items ? item[half] : -1;
            const int iu = tid % Y::U;
            float c_state[2] = {0.0f, 0.0f};
            // The projection's values come through shared memory, 16 bytes a thread: a load into registers one step ahead took
            // longer than the step (2500 cycles behind the shared-memory traffic of the multiplications), and every gate waited.
            const int fg = iu / (Y::U / 4), fu = iu % (Y::U / 4) * 4;           // gate and first unit that this thread fetches
            auto fetch = [&](int t, int half) {
                if (item[half] >= 0 && t < T) {
                    const int ir = item[half] / Y::U, row = b0 + half * RH + ir;
                    const float* p = pre + (static_cast<int64_t>(t) * B + (row < B ? row : 0)) * (4 * H) + fg * H + j0 + fu;
                    const uint32_t to = smem_u32(pre_s + (((t % (kRecAhead + 1)) * 2 + half) * Y::Items + item[half]) * 4);
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(p) : "memory");
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            pdl_wait();  // the projection; the weights are not its output
#pragma unroll
            for (int t = 0; t < kRecAhead; ++t) {
                fetch(t, 0);
                fetch(t, 1);
            }
            // this lane sends its quad of units to four CTAs
            uint32_t dst[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) dst[k] = map_remote(smem_u32(smem_raw), static_cast<uint32_t>((lane & 3) * 4 + k));
            const uint32_t h_off = smem_u32(h_s + rank * Y::BP) - smem_u32(smem_raw);
            const uint32_t bar_off = smem_u32(full) - smem_u32(smem_raw);
            cluster_wait();
#pragma unroll 1
            for (int t = 0; t < T; ++t) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    asm volatile("cp.async.wait_group %0;" ::"n"(2 * kRecAhead - 1) : "memory");
                    if (mine[half]) {
                        const int i = item[half] >= 0 ? item[half] : 0;
                        __syncwarp();
                        if (t > 0)  // the partial sums of all warps, the fetched values of all gate threads
                            asm volatile("barrier.sync %0, %1;" ::"r"(1 + half), "n"(kPairFma + Y::GateWarps * 32) : "memory");
                        else
                            asm volatile("barrier.sync %0, %1;" ::"r"(3 + half), "n"(Y::GateWarps * 32) : "memory");
                        const float* pre_t = pre_s + ((t % (kRecAhead + 1)) * 2 + half) * (Y::Items * 4) + i / Y::U * (4 * Y::U) + iu;
                        float gate[4];
#pragma unroll
                        for (int g = 0; g < 4; ++g) gate[g] = pre_t[g * Y::U];
                        if (t > 0) {
                            const float4* p = reinterpret_cast<const float4*>(part) + half * Y::KQ * Y::Items + i;
                            float4 s = p[0];
#pragma unroll
                            for (int k = 1; k < Y::KQ; ++k) {
                                const float4 v = p[k * Y::Items];
                                s.x = __fadd_rn(s.x, v.x);
                                s.y = __fadd_rn(s.y, v.y);
                                s.z = __fadd_rn(s.z, v.z);
                                s.w = __fadd_rn(s.w, v.w);
                            }
                            gate[0] = __fadd_rn(gate[0], s.x);
                            gate[1] = __fadd_rn(gate[1], s.y);
                            gate[2] = __fadd_rn(gate[2], s.z);
                            gate[3] = __fadd_rn(gate[3], s.w);
                        }
                        const bool sends = item[half] >= 0 && *late == 0;
                        float sg[3] = {gate[0], gate[1], gate[3]};
                        sigmoid_f32_n(sg);
                        const float ig = sg[0], fgt = sg[1], og = sg[2], gg = tanhf(gate[2]);
                        c_state[half] = __fadd_rn(__fmul_rn(fgt, c_state[half]), __fmul_rn(ig, gg));
                        const float hval = __fmul_rn(og, tanhf(c_state[half]));
                        if (t + 1 < T) {
                            float v[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) v[k] = __shfl_sync(kFullMask, hval, (lane & ~3) + k);
                            const uint32_t to = h_off + static_cast<uint32_t>((((t + 1) & 1) * 2 + half) * (kRecCluster * Y::BP) + (i & ~3)) * 4;
                            const uint32_t bar = bar_off + static_cast<uint32_t>(half * 2 + ((t + 1) & 1)) * 8;
                            if (sends) {
#pragma unroll
                                for (int k = 0; k < 4; ++k) store_async4(dst[k] + to, v[0], v[1], v[2], v[3], dst[k] + bar);
                            }
                        }
                        const int row = b0 + half * RH + i / Y::U;
                        if (item[half] >= 0 && row < B) {
                            const int64_t o = (static_cast<int64_t>(t) * B + row) * H + j0 + iu;
                            hs[o] = hval;
                            cs[o] = c_state[half];
                        }
                    }
                    fetch(t + kRecAhead, half);  // (into the place of step t - 1, which all threads have read)
                }
            }
        } else {
            cluster_wait();
        }
    }
    cluster_arrive();  // nobody leaves while another CTA may still store into its shared memory
    cluster_wait();
    if (*late) {       // (stores of h that nobody waited for may be under way; they arrive within microseconds)
        const unsigned long long t0 = clock64();
        while (clock64() - t0 < 400000ull) {
        }
    }
}

// A single step multiplies nothing: its gates, without a cluster that fetches weights and sets up an exchange.
constexpr int kFirstThreads = 128;
__global__ void __launch_bounds__(kFirstThreads)
lstm_first_step_kernel(const float* __restrict__ pre, int B, int H, float* __restrict__ hs, float* __restrict__ cs) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kFirstThreads + threadIdx.x;  // (row, unit)
    const int64_t row = i / H;
    pdl_wait();  // the projection (read with __ldcg: a __ldg could be moved up across this)
    if (row >= B) return;
    const float* p = pre + row * (4 * H) + (i - row * H);
    float sg[3] = {__ldcg(p), __ldcg(p + H), __ldcg(p + 3 * H)};
    const float gg = tanhf(__ldcg(p + 2 * H));
    sigmoid_f32_n(sg);
    const float c = __fadd_rn(__fmul_rn(sg[1], 0.0f), __fmul_rn(sg[0], gg));  // (a forget gate that is NaN stays one)
    hs[i] = __fmul_rn(sg[2], tanhf(c));
    cs[i] = c;
}

template <class... KP, class... A>
static int launch_rec(void (*kernel)(KP...), int threads, size_t smem, int rows, int B, bool after, cudaStream_t st, A... args) {
    FB_TRY(check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)), "lstm_recurrent attr"));
    FB_TRY(check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1), "lstm_recurrent attr"));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>((B + rows - 1) / rows) * kRecCluster);
    cfg.blockDim = dim3(static_cast<unsigned>(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kRecCluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // the weights are fetched while the projection ends
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = after ? 2 : 1;
    FB_TRY(check_cuda(cudaLaunchKernelEx(&cfg, kernel, static_cast<KP>(args)...), "lstm_recurrent launch"));
    count_launch();
    return FB_OK;
}
template <int H, int R>
static int launch_narrow(const float* pre, const float* w_hh, int T, int B, float* hs, float* cs, int32_t* status, cudaStream_t st) {
    static_assert(RecLayout<H, R>::bytes <= 227 * 1024, "shared memory of one CTA");
    return launch_rec(lstm_recurrent_kernel<H, R, 0>, kRecThreads, RecLayout<H, R>::bytes, R, B, true, st, pre, w_hh, T, B, hs, cs, status,
                      t_rec_drop, RecInput{});
}
template <int H, int R>
static int launch_pair(const float* pre, const float* w_hh, int T, int B, float* hs, float* cs, int32_t* status, cudaStream_t st) {
    using Y = PairLayout<H, R / 2>;
    static_assert(R % 2 == 0 && Y::bytes <= 227 * 1024, "shared memory of one CTA");
    return launch_rec(lstm_recurrent_pair_kernel<H, R / 2>, kPairThreads, Y::bytes, R, B, true, st, pre, w_hh, T, B, hs, cs, status, t_rec_drop);
}

// Rows per cluster: the fewest that let all clusters run at once (seven clusters of sixteen whole SMs fit a B200; more clusters
// than that run one after the other).
constexpr int kClusters = 7;
template <int H>
static int launch_rec_rows(const float* pre, const float* w_hh, int T, int B, float* hs, float* cs, int32_t* status, cudaStream_t st) {
    if (B <= kClusters) return launch_narrow<H, 1>(pre, w_hh, T, B, hs, cs, status, st);
    if (B <= 2 * kClusters) return launch_narrow<H, 2>(pre, w_hh, T, B, hs, cs, status, st);
    if (B <= 4 * kClusters) return launch_pair<H, 4>(pre, w_hh, T, B, hs, cs, status, st);
    if (B <= 6 * kClusters) return launch_pair<H, 6>(pre, w_hh, T, B, hs, cs, status, st);
    if (B <= 8 * kClusters) return launch_pair<H, 8>(pre, w_hh, T, B, hs, cs, status, st);
    return launch_pair<H, 10>(pre, w_hh, T, B, hs, cs, status, st);
}

int launch_lstm_recurrent(const float* pre, const float* w_hh, int T, int B, int H, float* hs, float* cs, int32_t* status, cudaStream_t st) {
    FB_REQUIRE(H == 256 || H == 512, "lstm recurrence: hidden size %d not supported (256 or 512)", H);
    if (T == 1) {
        const int64_t blocks = (static_cast<int64_t>(B) * H + kFirstThreads - 1) / kFirstThreads;
        return launch_after(lstm_first_step_kernel, dim3(static_cast<unsigned>(blocks)), dim3(kFirstThreads), 0, st, true, "lstm_first_step launch",
                            pre, B, H, hs, cs);
    }
    return H == 512 ? launch_rec_rows<512>(pre, w_hh, T, B, hs, cs, status, st) : launch_rec_rows<256>(pre, w_hh, T, B, hs, cs, status, st);
}

// ---- the whole call in one launch ----
bool lstm_one_launch(int T, int B, int K, int H) {
    const int rows = T * (B <= kClusters ? 1 : 2);
    return H == 256 && B <= 2 * kClusters && K <= 512 && T <= kOneLaunchSteps && rows <= kOneLaunchRows;
}
template <int R, int PQ>
static int launch_one(const RecInput& in, const float* w_hh, int T, int B, float* hs, float* cs, int32_t* status, cudaStream_t st) {
    return launch_rec(lstm_recurrent_kernel<256, R, PQ>, kRecThreads, ProjLayout<256, R, PQ>::bytes(T), R, B, false, st,
                      static_cast<const float*>(nullptr), w_hh, T, B, hs, cs, status, t_rec_drop, in);
}
template <int R>
static int launch_one_depth(const RecInput& in, const float* w_hh, int T, int B, float* hs, float* cs, int32_t* status, cudaStream_t st) {
    switch ((in.K + 127) / 128) {
        case 1: return launch_one<R, 1>(in, w_hh, T, B, hs, cs, status, st);
        case 2: return launch_one<R, 2>(in, w_hh, T, B, hs, cs, status, st);
        case 3: return launch_one<R, 3>(in, w_hh, T, B, hs, cs, status, st);
        default: return launch_one<R, 4>(in, w_hh, T, B, hs, cs, status, st);
    }
}
int launch_lstm_one(const float* x, const float* w_ih, const float* b_ih, const float* b_hh, const float* w_hh, int T, int B, int K, float* hs,
                    float* cs, int32_t* status, cudaStream_t st) {
    const RecInput in{x, w_ih, b_ih, b_hh, K};
    return B <= kClusters ? launch_one_depth<1>(in, w_hh, T, B, hs, cs, status, st) : launch_one_depth<2>(in, w_hh, T, B, hs, cs, status, st);
}

}  // namespace fb
