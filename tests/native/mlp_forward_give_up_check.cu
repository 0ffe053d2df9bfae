// The inference kernel when one thread gives up on the last chain of its warpgroup's last tile: its row is NaN
// and the status says so.  The give-up is a stand-in, nothing waits for its limit.
// Prints "plain <status> <NaN rows> given_up <status> <NaN rows> after <status> <NaN rows>".
#include <cstdio>
#include <cmath>
#include <vector>

__device__ int give_up_row = -1;
#define FT_GIVE_UP(k) ((k) + FT_WGS >= ktiles && (int)row_of(k) == give_up_row)
#include "sph_mlp.cu"

namespace wsph {
int set_error(int code, const char*, ...) { return code; }
int check_launch(const char*) { return cudaGetLastError() == cudaSuccess ? SPH_OK : SPH_ERR_CUDA; }
void count_launch() {}
}  // namespace wsph

#define CK(x) do { if ((x) != cudaSuccess) { fprintf(stderr, "%s: %s\n", #x, cudaGetErrorString(cudaGetLastError())); return 1; } } while (0)

int main() {
    const int64_t n = 148 * 128 * 2 + 37, np = sph_mlp_param_count();
    std::vector<float> theta(np), feats(n * 8), y(n);
    unsigned int r = 1u;
    auto rnd = [&] { r = r * 1664525u + 1013904223u; return (float)(r >> 8) / 8388608.f - 1.f; };
    for (float& v : theta) v = 0.2f * rnd();
    for (float& v : feats) v = rnd();
    float *t, *f, *out;
    int32_t* st;
    CK(cudaMalloc(&t, np * 4)); CK(cudaMalloc(&f, n * 32)); CK(cudaMalloc(&out, n * 4)); CK(cudaMalloc(&st, 4));
    CK(cudaMemcpy(t, theta.data(), np * 4, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(f, feats.data(), n * 32, cudaMemcpyHostToDevice));
    const int rows[3] = {-1, 148 * 128 + 5, -1};      // the second tile of block 0: the last of its warpgroup
    const char* names[3] = {"plain", "given_up", "after"};
    for (int k = 0; k < 3; ++k) {
        int32_t s = 0;
        CK(cudaMemcpyToSymbol(give_up_row, &rows[k], 4)); CK(cudaMemset(st, 0, 4)); CK(cudaMemset(out, 0, n * 4));
        if (sph_mlp_forward_tc(t, n, f, nullptr, out, st, nullptr) != SPH_OK) return 1;
        CK(cudaDeviceSynchronize());
        CK(cudaMemcpy(&s, st, 4, cudaMemcpyDeviceToHost)); CK(cudaMemcpy(y.data(), out, n * 4, cudaMemcpyDeviceToHost));
        int nans = 0;
        for (float v : y) nans += std::isnan(v);
        printf("%s %d %d ", names[k], s, nans);
    }
    printf("\n");
    return 0;
}
