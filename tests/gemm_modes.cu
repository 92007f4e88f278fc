// Every epilogue of the GEMM at ragged M and N, with rows that start on
// 32-byte boundaries (whole sectors per lane) and with rows that do not
// (through shared memory).  Inputs are small integers, so the sums are exact
// in fp32 and every output is compared for equality: fp32 as it is, bf16
// rounded to nearest.  What lies around the output is not written.  Built and
// run by tests/test_gpu_gemm_modes.py.
#include <cstdint>
#include <cstdio>
#include <vector>

#include "tc_gemm.cuh"

using bf16 = __nv_bfloat16;
static uint64_t rng = 0x6502;
static int small_int() {   // -8 .. 8
    uint64_t z = (rng += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return (int)((z >> 40) % 17) - 8;
}
static bool ok(cudaError_t e, const char* what) {
    if (e != cudaSuccess) std::printf("%s: %s\n", what, cudaGetErrorString(e));
    return e == cudaSuccess;
}
template <class T>
static T* up(const std::vector<T>& h) {
    T* d = nullptr;
    if (!ok(cudaMalloc((void**)&d, h.size() * sizeof(T)), "cudaMalloc") ||
        !ok(cudaMemcpy(d, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice), "cudaMemcpy")) std::exit(2);
    return d;
}
static std::vector<bf16> ints(size_t n) {
    std::vector<bf16> v(n);
    for (bf16& x : v) x = __float2bfloat16((float)small_int());
    return v;
}

int main() {
    if (!tcg::prepare_gemm()) { std::printf("prepare_gemm failed\n"); return 2; }
    const int K = 192, pad = 64;   // elements around the output, a multiple of 32 bytes
    int* err = up(std::vector<int>(1, 0));
    long cases = 0, bad = 0;
    for (int M : {1, 31, 33, 128, 200, 300})
        for (int N : {16, 40, 200, 208, 257, 512}) {
            const std::vector<bf16> a = ints((size_t)M * K), b = ints((size_t)N * K), act = ints((size_t)M * N + 2 * pad);
            std::vector<float> bias(N + 4), ref((size_t)M * N);
            for (float& x : bias) x = (float)small_int();
            for (int i = 0; i < M; i++)
                for (int j = 0; j < N; j++) {
                    float s = 0;
                    for (int k = 0; k < K; k++) s += __bfloat162float(a[(size_t)i * K + k]) * __bfloat162float(b[(size_t)j * K + k]);
                    ref[(size_t)i * N + j] = s;
                }
            bf16 *da = up(a), *db = up(b), *dact = up(act);
            float* dbias = up(bias);
            const size_t n = (size_t)M * N + 2 * pad;
            const std::vector<float> f0(n, 7.0f);
            const std::vector<bf16> h0(n, __float2bfloat16(7.0f));
            for (int mode : {tcg::EPI_F32, tcg::EPI_BIAS_F32, tcg::EPI_BIAS_RELU, tcg::EPI_RELU_GRAD})
                for (int off : {0, 1}) {
                    const bool f32 = mode == tcg::EPI_F32 || mode == tcg::EPI_BIAS_F32;
                    float* df = up(f0);
                    bf16* dh = up(h0);
                    tcg::Epilogue e{};
                    e.mode = mode;
                    e.out_f32 = df + pad + off;
                    e.out_bf16 = dh + pad + off;
                    e.bias = dbias + off;
                    e.act = dact + pad + off;
                    e.ldc = N;
                    int failed = 0;
                    std::vector<float> f(n);
                    std::vector<bf16> h(n);
                    if (!tcg::launch_gemm(da, K, db, K, M, N, K, e, err, nullptr) || !ok(cudaDeviceSynchronize(), "gemm") ||
                        !ok(cudaMemcpy(&failed, err, sizeof failed, cudaMemcpyDeviceToHost), "cudaMemcpy") || failed ||
                        !ok(cudaMemcpy(f.data(), df, n * sizeof(float), cudaMemcpyDeviceToHost), "cudaMemcpy") ||
                        !ok(cudaMemcpy(h.data(), dh, n * sizeof(bf16), cudaMemcpyDeviceToHost), "cudaMemcpy")) {
                        std::printf("M %d N %d mode %d: not run\n", M, N, mode);
                        return 2;
                    }
                    long wrong = 0;
                    for (size_t i = 0; i < n; i++) {
                        float want = 7.0f;
                        if (i >= (size_t)(pad + off) && i < (size_t)(pad + off) + ref.size()) {
                            const size_t o = i - pad - off;
                            want = ref[o];
                            if (mode == tcg::EPI_BIAS_F32 || mode == tcg::EPI_BIAS_RELU) want += bias[off + o % N];
                            if (mode == tcg::EPI_BIAS_RELU) want = want > 0 ? want : 0;
                            if (mode == tcg::EPI_RELU_GRAD) want = __bfloat162float(act[i]) > 0 ? want : 0;
                        }
                        wrong += f32 ? f[i] != want || __bfloat162float(h[i]) != 7.0f
                                     : __bfloat162float(h[i]) != __bfloat162float(__float2bfloat16(want)) || f[i] != 7.0f;
                    }
                    cases++;
                    if (wrong && bad++ < 20) std::printf("M %d N %d mode %d offset %d: %ld wrong\n", M, N, mode, off, wrong);
                    cudaFree(df);
                    cudaFree(dh);
                }
            cudaFree(da);
            cudaFree(db);
            cudaFree(dact);
            cudaFree(dbias);
        }
    std::printf("%ld cases, %ld wrong\n", cases, bad);
    return bad ? 1 : 0;
}
