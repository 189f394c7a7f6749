// The pair-once sum where a CTA gives up (test_pp_sym_gave_up_gpu.py): a plan whose
// one range meets more blocks than a CTA takes, which the kernel's own check
// reports. The outputs stay as they were, for that launch and for whole ones
// behind it, until the word is cleared; then they are the whole plan's again.
#include <cstdio>
#include <cstring>
#include <vector>

#include "pp_sym.cu"

using namespace nbody;

#define CK(x) do { const cudaError_t e_ = (x); if (e_ != cudaSuccess) { std::printf("%s: %s\n", #x, cudaGetErrorString(e_)); return 1; } } while (0)
#define CHECK(x) do { if (!(x)) { std::printf("FAILED: %s\n", #x); return 1; } } while (0)

int main() {
    const int64_t n = 5 * kSymB;
    cudaDeviceProp prop;
    CK(cudaGetDeviceProperties(&prop, 0));
    const SymPlan whole = pp_sym_plan(n, prop.multiProcessorCount);
    CHECK(whole.blocks == 5);
    SymPlan wide = whole;  // the same layout of parts and rows, one CTA for all tiles
    wide.ctas = 1;
    wide.begin[1] = whole.begin[whole.ctas];
    std::vector<float4> pos(n), out(n);
    for (int64_t i = 0; i < n; ++i)
        pos[i] = make_float4(static_cast<float>(i % 17), static_cast<float>(i % 101), static_cast<float>(i % 997), 1.f);
    float4 *dp, *df;
    char *scratch;
    int *status, h = 0;
    CK(cudaMalloc(&dp, n * sizeof(float4)));
    CK(cudaMalloc(&df, n * sizeof(float4)));
    CK(cudaMalloc(&scratch, 256 + whole.bytes));
    CK(cudaMalloc(&status, sizeof(int)));
    CK(cudaMemcpy(dp, pos.data(), n * sizeof(float4), cudaMemcpyHostToDevice));
    CK(cudaMemset(scratch, 0, 256 + whole.bytes));
    CK(cudaMemset(status, 0, sizeof(int)));
    Integrate g;
    g.force = df;
    const auto run = [&](const SymPlan &p) -> int {
        CK(cudaMemset(df, 0xff, n * sizeof(float4)));
        CK(pp_sym_launch(p, dp, n, 40.f, g, scratch + 256, nullptr, status));
        CK(cudaMemcpy(out.data(), df, n * sizeof(float4), cudaMemcpyDeviceToHost));
        CK(cudaMemcpy(&h, status, sizeof(int), cudaMemcpyDeviceToHost));
        return 0;
    };
    const auto untouched = [&] {
        for (const float4 &f : out) {
            unsigned bits[4];
            std::memcpy(bits, &f, sizeof(bits));
            for (unsigned b : bits)
                if (b != 0xffffffffu) return false;
        }
        return true;
    };
    if (run(whole)) return 1;
    CHECK(h == NBODY_OK);
    const std::vector<float4> want = out;
    CHECK(!untouched());
    if (run(wide)) return 1;
    CHECK(h == NBODY_ERR_CAPACITY);
    CHECK(untouched());
    if (run(whole)) return 1;
    CHECK(untouched());
    CK(cudaMemset(scratch, 0, 256));
    CK(cudaMemset(status, 0, sizeof(int)));
    if (run(whole)) return 1;
    CHECK(h == NBODY_OK && std::memcmp(out.data(), want.data(), n * sizeof(float4)) == 0);
    return 0;
}
