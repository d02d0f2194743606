// unb::reciprocal and unb::quotient on the GPU against the division of the
// same operands there and on the host, bit for bit: every exponent that a
// composite alpha or blend denominator may have, significands at both ends and
// random. Prints the number of differences.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>

#include "quotient.hpp"

__global__ void check(const double* a, const double* b, int n, double* r, double* q, int* differ) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = unb::reciprocal(b[i]);
    q[i] = unb::quotient(a[i], b[i], r[i]);
    if (r[i] != __drcp_rn(b[i]) || q[i] != __ddiv_rn(a[i], b[i])) atomicAdd(differ, 1);
}

int main() {
    uint64_t state = 0x9E3779B97F4A7C15ull;
    auto next = [&] { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; };
    auto make = [](uint64_t significand, int exponent) {
        const uint64_t u = (uint64_t(exponent + 1023) << 52) | (significand & 0xFFFFFFFFFFFFFull);
        double d;
        std::memcpy(&d, &u, 8);
        return d;
    };
    std::vector<double> a, b;
    for (int e = -40; e <= 240; ++e)
        for (int k = 0; k < 4096; ++k) {
            const uint64_t sig = k < 64 ? 0xFFFFFFFFFFFFFull - k : k < 128 ? uint64_t(k - 64) : next();
            b.push_back(make(sig, e));
            a.push_back(make(k % 3 ? next() : sig, int(next() % 101) - 60) * (k & 1 ? 1.0 : -1.0));
        }
    const int n = int(b.size());
    double *d_a, *d_b, *d_r, *d_q;
    int* d_n;
    const size_t bytes = size_t(n) * sizeof(double);
    int differ = 0;
    std::vector<double> r(n), q(n);
    bool ok = cudaMalloc(&d_a, bytes) == cudaSuccess && cudaMalloc(&d_b, bytes) == cudaSuccess &&
              cudaMalloc(&d_r, bytes) == cudaSuccess && cudaMalloc(&d_q, bytes) == cudaSuccess &&
              cudaMalloc(&d_n, sizeof(int)) == cudaSuccess &&
              cudaMemcpy(d_a, a.data(), bytes, cudaMemcpyHostToDevice) == cudaSuccess &&
              cudaMemcpy(d_b, b.data(), bytes, cudaMemcpyHostToDevice) == cudaSuccess &&
              cudaMemset(d_n, 0, sizeof(int)) == cudaSuccess;
    if (ok) check<<<(n + 255) / 256, 256>>>(d_a, d_b, n, d_r, d_q, d_n);
    ok = ok && cudaGetLastError() == cudaSuccess &&
         cudaMemcpy(&differ, d_n, sizeof(int), cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(r.data(), d_r, bytes, cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(q.data(), d_q, bytes, cudaMemcpyDeviceToHost) == cudaSuccess;
    if (!ok) {
        std::printf("CUDA call failed\n");
        return 2;
    }
    for (int i = 0; i < n; ++i)
        if (r[i] != 1.0 / b[i] || q[i] != a[i] / b[i]) ++differ;
    std::printf("%d of %d\n", differ, n);
    return differ ? 1 : 0;
}
