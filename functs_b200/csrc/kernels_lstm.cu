// C4: imperative LSTM (functs/benchmark/ai_model/lstm/lstm.py:79-98, 118-133) in two launches, or in one where a cluster of
// the recurrence has few rows (lstm_one_launch).
//
//   launch 1  input projection, hoisted out of the time loop because it does not depend on h:
//             pre[t*B + b, g*H + j] = x[t, b, :] @ w_ih[g, :, j] + b_ih[g, j] + b_hh[g, j]
//             (tensor cores: see kernels_lstm_tc.cu; the fp32 CUDA-core GEMM below is the device-side check)
//   launch 2  the whole recurrence (kernels_lstm_rec.cu; on the tensor cores, mode 2: kernels_lstm_tc.cu)
#include <cstring>

#include "common.cuh"

namespace fb {

int launch_lstm_input_proj_tc(const float* x, const float* w_ih, const float* b_ih, const float* b_hh, int M, int K,
                              int H, float* pre, void* tc_scratch, int32_t* status, cudaStream_t st);  // kernels_lstm_tc.cu
int64_t lstm_tc_scratch_bytes(int M, int K, int H);
bool lstm_tc_supported(int M, int K, int H);
bool lstm_rtc_supported(int B, int H);
int64_t lstm_rtc_scratch_bytes(int H);
int launch_lstm_recurrent(const float* pre, const float* w_hh, int T, int B, int H, float* hs, float* cs, int32_t* status, cudaStream_t st);  // kernels_lstm_rec.cu
bool lstm_one_launch(int T, int B, int K, int H);
int launch_lstm_one(const float* x, const float* w_ih, const float* b_ih, const float* b_hh, const float* w_hh, int T, int B, int K, float* hs,
                    float* cs, int32_t* status, cudaStream_t st);
int launch_lstm_recurrent_tc(const float* pre, const float* w_hh, int T, int B, int H, float* hs, float* cs, void* h_tiles,
                             unsigned int* step_counter, int32_t* status, cudaStream_t st);

// ---- fp32 CUDA-core GEMM with bias (check path for launch 1) ------------------------------------------------
constexpr int kGemmBM = 64, kGemmBN = 64, kGemmBK = 16;

__global__ void __launch_bounds__(256)
lstm_input_proj_simt_kernel(const float* __restrict__ x, const float* __restrict__ w_ih, const float* __restrict__ b_ih,
                            const float* __restrict__ b_hh, int M, int K, int H, float* __restrict__ pre) {
    __shared__ float As[kGemmBK][kGemmBM + 4];
    __shared__ float Bs[kGemmBK][kGemmBN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * kGemmBM;
    const int n0 = blockIdx.x * kGemmBN;  // column in [0, 4H); a tile never straddles two gates (H % 64 == 0)
    const int g = n0 / H, j0 = n0 - g * H;
    const float* __restrict__ Bg = w_ih + static_cast<int64_t>(g) * K * H;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += kGemmBK) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e = threadIdx.x + r * 256;  // 0..1023
            const int am = e >> 4, ak = e & 15;   // A tile: 64 rows x 16 k
            const int gm = m0 + am, gk = k0 + ak;
            As[ak][am] = (gm < M && gk < K) ? __ldg(x + static_cast<int64_t>(gm) * K + gk) : 0.0f;
            const int bk = e >> 6, bn = e & 63;   // B tile: 16 k x 64 cols
            const int gk2 = k0 + bk;
            Bs[bk][bn] = (gk2 < K) ? __ldg(Bg + static_cast<int64_t>(gk2) * H + j0 + bn) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kGemmBK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int jj = j0 + tx * 4 + j;
            const float bias = __fadd_rn(__ldg(b_ih + g * H + jj), __ldg(b_hh + g * H + jj));
            pre[static_cast<int64_t>(gm) * (4 * H) + g * H + jj] = __fadd_rn(acc[i][j], bias);
        }
    }
}

static inline int64_t align_up(int64_t v, int64_t a) { return (v + a - 1) / a * a; }

// what mode 0 means beyond the one launch: the combination measured fastest at T = 64, B = 64, H = 512
constexpr int kLstmDefaultMode = 3;

}  // namespace fb

namespace fb {
void yolo_set_prune(int on);
void lstm_set_drop_exchange(int on);
}

extern "C" {

int64_t functs_b200_lstm_scratch_bytes(int32_t seq_len, int32_t batch, int32_t input, int32_t hidden) {
    if (seq_len <= 0 || batch <= 0 || input <= 0 || hidden <= 0) return 0;
    const int64_t M = static_cast<int64_t>(seq_len) * batch;
    int64_t total = 256;                                             // step counter
    total += fb::align_up(M * 4 * hidden * 4, 256);                  // pre-activations from the input projection
    total += fb::align_up(fb::lstm_tc_scratch_bytes(static_cast<int>(M), input, hidden), 256);
    total += fb::align_up(fb::lstm_rtc_scratch_bytes(hidden), 256);  // h tiles of the tensor-core recurrence
    return total;
}

// mode: 0 = default; 1 = fp32 CUDA cores for both GEMMs; 2 = tensor cores for both (where the shapes allow it);
//       3 = tensor-core projection + CUDA-core recurrence
int functs_b200_lstm_forward_mode(const float* x, const float* w_ih, const float* w_hh, const float* b_ih,
                                  const float* b_hh, int32_t seq_len, int32_t batch, int32_t input, int32_t hidden,
                                  float* hs, float* cs, int32_t* status, void* scratch, void* stream, int32_t mode) {
    using namespace fb;
    FB_REQUIRE(x && w_ih && w_hh && b_ih && b_hh && hs && cs && scratch, "lstm_forward: null pointer");
    FB_REQUIRE(seq_len > 0 && batch > 0 && input > 0, "lstm_forward: bad sizes");
    FB_REQUIRE(hidden == 256 || hidden == 512, "lstm_forward: hidden size %d not supported (256 or 512)", hidden);
    FB_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 255) == 0 && (reinterpret_cast<uintptr_t>(hs) & 15) == 0,
               "lstm_forward: scratch must be 256-byte aligned and hs 16-byte aligned");
    cudaStream_t st = as_stream(stream);
    const int M = seq_len * batch;
    unsigned char* base = static_cast<unsigned char*>(scratch);
    unsigned int* counter = reinterpret_cast<unsigned int*>(base);
    float* pre = reinterpret_cast<float*>(base + 256);
    void* tc_scratch = base + 256 + align_up(static_cast<int64_t>(M) * 4 * hidden * 4, 256);
    void* rtc_scratch = static_cast<unsigned char*>(tc_scratch) + align_up(lstm_tc_scratch_bytes(M, input, hidden), 256);
    FB_REQUIRE(mode >= 0 && mode <= 3, "lstm_forward: mode %d unknown", mode);
    record_stage_event(0, st);
    if (mode == 0 && lstm_one_launch(seq_len, batch, input, hidden)) {
        record_stage_event(1, st);
        const int rc = launch_lstm_one(x, w_ih, b_ih, b_hh, w_hh, seq_len, batch, input, hs, cs, status, st);
        record_stage_event(2, st);
        return rc;
    }
    if (mode == 0) mode = kLstmDefaultMode;
    if (mode != 1 && lstm_tc_supported(M, input, hidden)) {
        FB_TRY(launch_lstm_input_proj_tc(x, w_ih, b_ih, b_hh, M, input, hidden, pre, tc_scratch, status, st));
    } else {
        dim3 grid(4 * hidden / kGemmBN, (M + kGemmBM - 1) / kGemmBM);
        lstm_input_proj_simt_kernel<<<grid, 256, 0, st>>>(x, w_ih, b_ih, b_hh, M, input, hidden, pre);
        count_launch();
        FB_TRY(check_launch("lstm_input_proj_simt_kernel"));
    }

    record_stage_event(1, st);
    if (mode == 2 && lstm_rtc_supported(batch, hidden)) {
        FB_TRY(check_cuda(cudaMemsetAsync(counter, 0, 256, st), "memset step counter"));
        const int rc = launch_lstm_recurrent_tc(pre, w_hh, seq_len, batch, hidden, hs, cs, rtc_scratch, counter, status, st);
        record_stage_event(2, st);
        return rc;
    }
    FB_TRY(launch_lstm_recurrent(pre, w_hh, seq_len, batch, hidden, hs, cs, status, st));
    record_stage_event(2, st);
    return FB_OK;
}

int functs_b200_debug_set(const char* name, int32_t value) {
    if (name != nullptr && std::strcmp(name, "yolo_prune") == 0) {
        fb::yolo_set_prune(value);
        return FB_OK;
    }
    if (name != nullptr && std::strcmp(name, "lstm_drop_exchange") == 0) {
        fb::lstm_set_drop_exchange(value);
        return FB_OK;
    }
    fb::set_error("debug_set: unknown switch");
    return FB_ERR_NOT_FOUND;
}

int functs_b200_lstm_forward(const float* x, const float* w_ih, const float* w_hh, const float* b_ih,
                             const float* b_hh, int32_t seq_len, int32_t batch, int32_t input, int32_t hidden,
                             float* hs, float* cs, int32_t* status, void* scratch, void* stream) {
    return functs_b200_lstm_forward_mode(x, w_ih, w_hh, b_ih, b_hh, seq_len, batch, input, hidden, hs, cs, status,
                                         scratch, stream, 0);
}

}  // extern "C"
