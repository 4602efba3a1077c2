// Test-only kernels: the arithmetic that leaves out rare repairs, and how often its permutations have to be run again.
#include "poseidon2_linear.cuh"
#include "gl_monolith.cuh"

namespace {
// row i of z: z0 .. z4 and the largest z4 that the caller allows for; out: the reduced word, whether a repair was told of
__global__ void reduce_kernel(const uint32_t* z, uint64_t* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t* p = z + 6 * i;
    gl::fast::Missed missed{0, 0};
    out[2 * i] = gl::fast::reduce(p[0], p[1], p[2], p[3], p[4], missed);
    out[2 * i + 1] = missed.any(p[5]);
}
// row i of s: a, b, c of a sum of words
__global__ void sum_kernel(const uint32_t* s, uint64_t* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    gl::fast::Missed missed{0, 0};
    out[2 * i] = gl::fast::reduce(gl::fast::Sum{s[3 * i], s[3 * i + 1], s[3 * i + 2]}, missed);
    out[2 * i + 1] = missed.any();
}
// count[0]: permutations of n states that the throughput form gives up; count[1]: words that differ from the exact form's, of the others
template <int W>
__global__ void permute_kernel(const uint64_t* states, int n, unsigned* count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t fast[W], exact[W];
    for (int j = 0; j < W; j++) fast[j] = exact[j] = states[(size_t)W * i + j];
    bool ok;
    if constexpr (W == 8) {
        ok = gl::poseidon2_permute_throughput(fast);
        gl::poseidon2_permute(exact);
    } else {
        ok = gl::monolith_permute_throughput(fast);
        gl::monolith_permute(exact);
    }
    if (!ok) atomicAdd(count, 1u);
    for (int j = 0; ok && j < W; j++)
        if (gl::canon(fast[j]) != gl::canon(exact[j])) atomicAdd(count + 1, 1u);
}
int done() { return cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess ? 0 : -1; }
}  // namespace

extern "C" {
int mc_reduce(const uint32_t* z, uint64_t* out, int n) {
    reduce_kernel<<<(n + 255) / 256, 256>>>(z, out, n);
    return done();
}
int mc_sum(const uint32_t* s, uint64_t* out, int n) {
    sum_kernel<<<(n + 255) / 256, 256>>>(s, out, n);
    return done();
}
int mc_permute(int width, const uint64_t* states, int n, unsigned* count) {
    if (width == 8) permute_kernel<8><<<(n + 127) / 128, 128>>>(states, n, count);
    else permute_kernel<12><<<(n + 127) / 128, 128>>>(states, n, count);
    return done();
}
}
