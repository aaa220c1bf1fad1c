// Generic fusion group without branches: one launch for a program that the host has cut into regions (program format:
// include/functs_b200.h, functs_b200_rprogram).  kernels_generic.cu evaluates the branches per element instead and serves the
// groups that cannot be cut.
//
// What bounded the interpreter there was issue (150 instructions per element of the channel-swap normalisation, most of them
// predicates, index arithmetic and decoding) and, for small groups, a chain of loads each waiting for the one before (11 us for
// 12 000 elements).  With the branches gone at the host:
//   - large outputs: a thread takes several elements of a region through each instruction, decoding it once; regions that
//     interleave (one per channel) are computed by the same CTA and stored through shared memory as whole runs, since a
//     store with stride R reaches every sector R times;
//   - small outputs: one element per thread, and all loads of the region's program are issued together before the first
//     instruction.
#include <algorithm>

#include "generic.cuh"
#include "region_plan.h"

namespace fb {

constexpr int kRegionSmall = 128;      // threads of the small form
constexpr int kRegionMaxInterleave = 8;

template <int R>
__device__ __forceinline__ void r_index(const functs_b200_region& G, int i, int (&y)[R]) {
    if (R == 1) {
        y[0] = i;
        return;
    }
    uint32_t rem = static_cast<uint32_t>(i);
#pragma unroll
    for (int k = R - 1; k >= 0; --k) {
        y[k] = 0;
        if (k < G.rank) {
            if (G.shape[k] > 1) {
                const uint32_t hi = __umulhi(G.div_magic[k], rem);
                const uint32_t q = (((rem - hi) >> 1) + hi) >> G.div_shift[k];
                y[k] = static_cast<int>(rem - q * static_cast<uint32_t>(G.shape[k]));
                rem = q;
            }
        }
    }
}
template <int R>
__device__ __forceinline__ int r_offset(int base, const int32_t (&coef)[4], const int (&y)[R]) {
    int o = base;
#pragma unroll
    for (int k = 0; k < R; ++k) o += coef[k] * y[k];
    return o;
}

// One instruction on V values; `fetch(l, v)` gives value v of load l.  Returns false at END.
template <int V, class Fetch>
__device__ __forceinline__ bool r_step(const functs_b200_ginstr I, float (&tos)[V], float (&st)[FB_G_STACK][V], int& sp, Fetch fetch) {
#define FB_R_EACH(expr)                                 \
    {                                                   \
        _Pragma("unroll") for (int v = 0; v < V; ++v) { \
            const float a = tos[v];                     \
            tos[v] = (expr);                            \
        }                                               \
        break;                                          \
    }
    switch (I.op) {
        case FB_G_END: return false;
        case FB_G_LOAD:
        case FB_G_CONST: {
            if (sp > 0) {
#pragma unroll
                for (int v = 0; v < V; ++v) st[sp - 1][v] = tos[v];
            }
            ++sp;
            if (I.op == FB_G_CONST) {
#pragma unroll
                for (int v = 0; v < V; ++v) tos[v] = I.imm.f;
            } else {
                fetch(I.arg, tos);
            }
            break;
        }
        // the common operators, one case each so that the switch is taken once for the V values
        case FB_G_ADD + FB_G_IMM: FB_R_EACH(__fadd_rn(a, I.imm.f))
        case FB_G_SUB + FB_G_IMM: FB_R_EACH(__fsub_rn(a, I.imm.f))
        case FB_G_MUL + FB_G_IMM: FB_R_EACH(__fmul_rn(a, I.imm.f))
        case FB_G_ADD: --sp; FB_R_EACH(__fadd_rn(st[sp - 1][v], a))
        case FB_G_SUB: --sp; FB_R_EACH(__fsub_rn(st[sp - 1][v], a))
        case FB_G_MUL: --sp; FB_R_EACH(__fmul_rn(st[sp - 1][v], a))
        case FB_G_EXP: FB_R_EACH(expf(a))
        case FB_G_SIGMOID: FB_R_EACH(sigmoid_f32(a))
        default: {
            const int op = I.op;
            if (op < FB_G_ADD) {
                FB_R_EACH(g_unary(op, a, I.imm.f))
            } else if (op < FB_G_ADD + FB_G_IMM) {
                --sp;
                FB_R_EACH(g_binary(op, st[sp - 1][v], a))
            } else if (op == FB_G_RSUB_IMM) {
                FB_R_EACH(__fsub_rn(I.imm.f, a))
            } else if (op == FB_G_RDIV_IMM) {
                FB_R_EACH(__fdiv_rn(I.imm.f, a))
            } else {
                FB_R_EACH(g_binary(op - FB_G_IMM, a, I.imm.f))
            }
        }
    }
#undef FB_R_EACH
    return true;
}

// Large form.  grid = (blocks of 256 * V elements of a region, regions), or with INTERLEAVE (blocks) and all regions per CTA.
// Dynamic shared memory: s_out (INTERLEAVE), then V floats per thread for each load that is fetched ahead (AHEAD): all loads of
// the CTA are on their way before the first instruction, instead of one instruction's at a time.  WINDOW: all loads step through
// one tensor as the output is stepped through (an element of every pixel, whatever its place in it), so the CTA's share of it is one
// run, fetched in 16-byte pieces; an element at a time, every line went through the load path once per region and word.
template <int R, bool INTERLEAVE, int FETCH>
__global__ void __launch_bounds__(kRegionThreads) region_group_kernel(const __grid_constant__ functs_b200_rprogram P) {
    constexpr bool AHEAD = FETCH == kAhead, WINDOW = FETCH == kWindow;
    static_assert(!WINDOW || (R == 1 && INTERLEAVE), "one run");
    constexpr int V = kRegionVec;
    extern __shared__ __align__(16) float s_region[];
    float* s_out = s_region;
    float* s_val = s_region + (INTERLEAVE ? P.interleave * kRegionThreads * V : 0);
    const int i0 = blockIdx.x * (kRegionThreads * V), t = threadIdx.x;
    const int r_begin = INTERLEAVE ? 0 : blockIdx.y, r_end = INTERLEAVE ? P.num_regions : r_begin + 1;
    if (AHEAD) {
        int slot = 0;
#pragma unroll 1
        for (int r = r_begin; r < r_end; ++r) {
            const functs_b200_region& G = P.region[r];
            if (i0 >= G.count) break;  // (interleaved regions have the same count)
            int y[V][R];
#pragma unroll
            for (int v = 0; v < V; ++v) r_index<R>(G, min(i0 + v * kRegionThreads + t, G.count - 1), y[v]);
#pragma unroll 1
            for (int l = G.first_load; l < G.first_load + G.num_loads; ++l, ++slot) {
                const functs_b200_rload& L = P.load[l];
                const float* p = static_cast<const float*>(P.in_ptr[L.tensor]);
                const uint32_t dst = smem_u32(s_val + slot * (kRegionThreads * V) + t);
#pragma unroll
                for (int v = 0; v < V; ++v)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + v * kRegionThreads * 4), "l"(p + r_offset<R>(L.base, L.coef, y[v]))
                                 : "memory");
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");  // a thread reads only what it has fetched itself
    }
    if (WINDOW) {
        const float* p = static_cast<const float*>(P.in_ptr[P.load[0].tensor]) + i0 * P.interleave;
        int n = kRegionThreads * V * P.interleave;
        if (i0 + kRegionThreads * V >= P.region[0].count) {  // the last CTA: no further than the loads reach
            int last = 0;
            for (int l = 0; l < P.num_loads; ++l) last = max(last, P.load[l].base);
            n = region_run_words(P.interleave, P.region[0].count - i0, last);
        }
        const int n4 = (reinterpret_cast<uintptr_t>(p) & 15) == 0 ? n >> 2 : 0;
        for (int i = t; i < n4; i += kRegionThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(s_val + 4 * i)), "l"(p + 4 * i) : "memory");
        for (int i = 4 * n4 + t; i < n; i += kRegionThreads)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(s_val + i)), "l"(p + i) : "memory");
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    int slot0 = 0;  // of the region's first load
#pragma unroll 1
    for (int r = r_begin; r < r_end; ++r) {
        const functs_b200_region& G = P.region[r];
        if (i0 >= G.count) break;
        int y[V][R];
#pragma unroll
        for (int v = 0; v < V; ++v) r_index<R>(G, min(i0 + v * kRegionThreads + t, G.count - 1), y[v]);
        float tos[V], st[FB_G_STACK][V];
        int sp = 0;
        auto fetch = [&](int l, float (&out)[V]) {
            if (AHEAD) {
#pragma unroll
                for (int v = 0; v < V; ++v) out[v] = s_val[(slot0 + l - G.first_load) * (kRegionThreads * V) + v * kRegionThreads + t];
                return;
            }
            const functs_b200_rload& L = P.load[l];
            if (WINDOW) {
#pragma unroll
                for (int v = 0; v < V; ++v) out[v] = s_val[(y[v][0] - i0) * P.interleave + L.base];
                return;
            }
            const void* p = P.in_ptr[L.tensor];
#pragma unroll
            for (int v = 0; v < V; ++v) out[v] = g_fetch(p, L.dtype, r_offset<R>(L.base, L.coef, y[v]));
        };
#pragma unroll 1
        for (int pc = G.first_instr; r_step<V>(P.instr[pc], tos, st, sp, fetch); ++pc) {
        }
        slot0 += G.num_loads;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const int i = v * kRegionThreads + t;
            if (INTERLEAVE) {
                s_out[i * P.interleave + G.out_base] = tos[v];
            } else if (i0 + i < G.count) {
                const int o = r_offset<R>(G.out_base, G.out_coef, y[v]);
                if (P.out_dtype == 0) static_cast<float*>(P.out_ptr)[o] = tos[v];
                else static_cast<uint8_t*>(P.out_ptr)[o] = tos[v] != 0.0f ? 1 : 0;
            }
        }
    }
    if (INTERLEAVE) {
        __syncthreads();
        const int first = i0 * P.interleave, n = min(kRegionThreads * V * P.interleave, P.numel - first);
        float* out = static_cast<float*>(P.out_ptr) + first;  // a multiple of 16 bytes behind out_ptr
        const int n4 = (reinterpret_cast<uintptr_t>(out) & 15) == 0 ? n >> 2 : 0;
        for (int i = t; i < n4; i += kRegionThreads) reinterpret_cast<float4*>(out)[i] = reinterpret_cast<const float4*>(s_out)[i];
        for (int i = 4 * n4 + t; i < n; i += kRegionThreads) out[i] = s_out[i];
    }
}

// Small form: one element per thread, the region's loads issued eight at a time before the program runs.
__global__ void __launch_bounds__(kRegionSmall) region_group_kernel_small(const __grid_constant__ functs_b200_rprogram P) {
    __shared__ float s_val[FB_R_REGION_LOADS][kRegionSmall];
    const functs_b200_region& G = P.region[blockIdx.y];
    const int i = blockIdx.x * kRegionSmall + threadIdx.x, t = threadIdx.x;
    if (i >= G.count) return;
    int y[4];
    r_index<4>(G, i, y);
#pragma unroll 1
    for (int l0 = 0; l0 < G.num_loads; l0 += 8) {
        float x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (l0 + u >= G.num_loads) break;
            const functs_b200_rload& L = P.load[G.first_load + l0 + u];
            x[u] = g_fetch(P.in_ptr[L.tensor], L.dtype, r_offset<4>(L.base, L.coef, y));
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (l0 + u < G.num_loads) s_val[l0 + u][t] = x[u];
    }
    float tos[1], st[FB_G_STACK][1];
    int sp = 0;
    auto fetch = [&](int l, float (&out)[1]) { out[0] = s_val[l - G.first_load][t]; };
#pragma unroll 1
    for (int pc = G.first_instr; r_step<1>(P.instr[pc], tos, st, sp, fetch); ++pc) {
    }
    const int o = r_offset<4>(G.out_base, G.out_coef, y);
    if (P.out_dtype == 0) static_cast<float*>(P.out_ptr)[o] = tos[0];
    else static_cast<uint8_t*>(P.out_ptr)[o] = tos[0] != 0.0f ? 1 : 0;
}

// Everything the kernels index with is checked here, so that they need no checks of their own.
static int validate(const functs_b200_rprogram& P) {
    FB_REQUIRE(P.num_regions > 0 && P.num_regions <= FB_R_MAX_REGIONS && P.num_instr > 0 && P.num_instr <= FB_R_MAX_INSTR &&
                   P.num_loads >= 0 && P.num_loads <= FB_R_MAX_LOADS && P.numel > 0 && P.out_ptr != nullptr,
               "region group: bad program header");
    for (int l = 0; l < P.num_loads; ++l) {
        const functs_b200_rload& L = P.load[l];
        FB_REQUIRE(L.tensor >= 0 && L.tensor < FB_G_MAX_INPUTS && P.in_ptr[L.tensor] != nullptr && L.dtype >= 0 && L.dtype <= 3,
                   "region group: bad load");
    }
    int64_t total = 0;
    for (int r = 0; r < P.num_regions; ++r) {
        const functs_b200_region& G = P.region[r];
        FB_REQUIRE(G.rank >= 1 && G.rank <= 4 && G.count > 0, "region group: bad region");
        int64_t n = 1, top = G.out_base;
        for (int k = 0; k < G.rank; ++k) {
            FB_REQUIRE(G.shape[k] > 0 && G.out_coef[k] >= 0 && (G.shape[k] == 1 || G.div_shift[k] < 32), "region group: bad extent");
            n *= G.shape[k];
            top += static_cast<int64_t>(G.out_coef[k]) * (G.shape[k] - 1);
        }
        FB_REQUIRE(n == G.count && G.out_base >= 0 && top < P.numel, "region group: a region leaves the output");
        total += n;
        FB_REQUIRE(G.first_load >= 0 && G.num_loads >= 0 && G.num_loads <= FB_R_REGION_LOADS && G.first_load + G.num_loads <= P.num_loads,
                   "region group: bad load range");
        if (P.interleave > 1) {
            int64_t run = P.interleave;
            for (int k = G.rank - 1; k >= 0; --k) {
                FB_REQUIRE(G.shape[k] == 1 || G.out_coef[k] == run, "region group: bad interleave");
                run *= G.shape[k];
            }
            FB_REQUIRE(G.out_base < P.interleave && G.count == P.region[0].count, "region group: bad interleave");
        }
        int depth = 0, pc = G.first_instr;
        FB_REQUIRE(pc >= 0, "region group: bad program");
        for (;; ++pc) {
            FB_REQUIRE(pc < P.num_instr, "region group: a program without an end");
            const functs_b200_ginstr& I = P.instr[pc];
            const int op = I.op;
            if (op == FB_G_END) break;
            if (op == FB_G_LOAD) FB_REQUIRE(I.arg >= G.first_load && I.arg < G.first_load + G.num_loads, "region group: load slot out of range");
            if (op == FB_G_LOAD || op == FB_G_CONST) {
                ++depth;
                FB_REQUIRE(depth <= FB_G_STACK, "region group: value stack too deep");
            } else if (op >= FB_G_ADD && op <= FB_G_NE) {
                --depth;
                FB_REQUIRE(depth >= 1, "region group: binary operator needs two values");
            } else {
                FB_REQUIRE(depth >= 1 && ((op >= FB_G_EXP && op <= FB_G_LOG) || (op >= FB_G_ADD + FB_G_IMM && op <= FB_G_NE + FB_G_IMM) ||
                                          op == FB_G_RSUB_IMM || op == FB_G_RDIV_IMM),
                           "region group: unknown instruction %d", op);
            }
        }
        FB_REQUIRE(depth == 1, "region group: the program must leave exactly one value");
    }
    FB_REQUIRE(total == P.numel && P.interleave <= kRegionMaxInterleave && (P.interleave <= 1 || (P.interleave == P.num_regions && P.out_dtype == 0)),
               "region group: the regions do not tile the output");
    return FB_OK;
}

}  // namespace fb

extern "C" int functs_b200_region_group_launch(const functs_b200_rprogram* program, void* stream) {
    using namespace fb;
    FB_REQUIRE(program != nullptr, "region group: null program");
    const functs_b200_rprogram& P = *program;
    FB_TRY(validate(P));
    cudaStream_t st = as_stream(stream);
    int most = 0, rank = 1;
    for (int r = 0; r < P.num_regions; ++r) {
        most = std::max(most, P.region[r].count);
        rank = std::max(rank, P.region[r].rank);
    }
    // Several elements per thread once that still makes two CTAs per SM; all regions in one CTA only where that leaves four per SM
    // (200 000 boxes decoded in four regions: 36 us with 195 CTAs that do all four, 14 us with one region per CTA, 25 us with one
    // element per thread).
    const bool inter = P.interleave > 1 && most >= kNumSMs * 4 * kRegionThreads * kRegionVec;
    if (P.numel < kNumSMs * 2 * kRegionThreads * kRegionVec) {
        const dim3 grid(static_cast<unsigned>((most + kRegionSmall - 1) / kRegionSmall), static_cast<unsigned>(P.num_regions));
        region_group_kernel_small<<<grid, kRegionSmall, 0, st>>>(P);
    } else {
        const unsigned blocks = static_cast<unsigned>((most + kRegionThreads * kRegionVec - 1) / (kRegionThreads * kRegionVec));
        const RegionPlan plan = region_plan(P, rank, inter);
        const dim3 grid(blocks, inter ? 1u : static_cast<unsigned>(P.num_regions));
        auto run = [&](auto k) { k<<<grid, kRegionThreads, plan.shared, st>>>(P); };
        auto by_rank = [&](auto kernel_rank1, auto kernel_rank2, auto kernel_rank4) {
            run(rank == 1 ? kernel_rank1 : rank == 2 ? kernel_rank2 : kernel_rank4);
        };
        if (plan.fetch == kWindow) run(region_group_kernel<1, true, kWindow>);
        else if (plan.fetch == kAhead) by_rank(region_group_kernel<1, true, kAhead>, region_group_kernel<2, true, kAhead>, region_group_kernel<4, true, kAhead>);
        else if (inter) by_rank(region_group_kernel<1, true, kEach>, region_group_kernel<2, true, kEach>, region_group_kernel<4, true, kEach>);
        else by_rank(region_group_kernel<1, false, kEach>, region_group_kernel<2, false, kEach>, region_group_kernel<4, false, kEach>);
    }
    count_launch();
    return check_launch("region_group_kernel");
}
