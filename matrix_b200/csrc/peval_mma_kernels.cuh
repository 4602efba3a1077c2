// First pass of a partial evaluation of a base-field table on the tensor cores: every row of 2^k elements dotted with the eq
// vector of k challenges, out[row] = sum_x in[2^k row + x] eq(r, x).
//
// The products of a row are a contraction of exact integers over the row's bytes as they lie in memory (pair_mma_kernels.cuh:
// the other operand holds the bytes of 2^(8 i) eq(x) mod p, sixteen 32-bit sums a row come back), so what is left is the
// traffic: 128 rows a tile, 256 bytes of each row a stage, three stages in flight. A block keeps the operand of at most 2^10
// elements (128 KB); longer rows are shared by the blocks of a cluster, which add their sums through each other's shared
// memory. On the integer pipes the two multiply-accumulates an element take 48 cycles a warp:
// whole calls, us, there / here: 2^22 elements, rows of 2^6 41 / 34, 2^9 49 / 38; 2^24, 2^6 71 / 51, 2^9 79 / 55, 2^12 70 / 57;
// 2^26, 2^6 175 / 120, 2^12 166 / 134.
#pragma once
#include "pair_mma_kernels.cuh"

namespace mb {
namespace pe {

constexpr int DM_BLK = 256, DM_ROWS = 128, DM_SLICE = 10, DM_MIN = 6, DM_MAX = 12;   // log2 of a block's, a row's elements
constexpr int DM_STAGES = 3;
constexpr uint32_t DM_STAGE = DM_ROWS * 256;
// stages, operand, and the small things: everything in dynamic shared memory, whose base is aligned to 64 bytes at least, so that
// with 960 bytes to align it to 1024 the longest operand just fits
constexpr uint32_t DM_EXTRA = DM_ROWS * 16 + 64;
__host__ __device__ constexpr uint32_t dm_smem(int k) { return DM_STAGES * DM_STAGE + (128u << (k < DM_SLICE ? k : DM_SLICE)) + DM_EXTRA + 960; }
static_assert(dm_smem(DM_MAX) <= 232448, "227 KB a block");

template <class FOut> struct DotField;
template <> struct DotField<sc::GlExt2> { using F = pr::GlF; };
template <> struct DotField<sc::AglExt2> { using F = pr::AglF; };

// words f[0 .. 8) -> words whose byte i is byte b of f[i]
__device__ __forceinline__ void transpose_bytes(const uint64_t (&f)[8], uint64_t (&o)[8]) {
#pragma unroll
    for (int half = 0; half < 2; half++) {      // bytes 0 .. 3 and 4 .. 7 of the words
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; i++) w[i] = half ? gl::hi32(f[i]) : gl::lo32(f[i]);
#pragma unroll
        for (int b = 0; b < 4; b++) {
            const uint32_t sel = b | ((4 + b) << 4);
            const uint32_t lo = __byte_perm(__byte_perm(w[0], w[1], sel), __byte_perm(w[2], w[3], sel), 0x5410);
            const uint32_t hi = __byte_perm(__byte_perm(w[4], w[5], sel), __byte_perm(w[6], w[7], sel), 0x5410);
            o[4 * half + b] = gl::pack64(lo, hi);
        }
    }
}

// A row without the tensor cores, from the operand (bytes of eq(x) are its bytes for i = 0): after a wait that ran out.
template <class F>
static __device__ __noinline__ typename F::E2 plain_row(const uint64_t* in, const uint8_t* op, int n) {
    using M = pr::MmaField<F>;
    typename F::E2 e{0, 0};
    for (int x = 0; x < n; x++) {
        uint64_t c[2] = {0, 0};
        for (int j = 0; j < 16; j++)
            c[j >> 3] |= (uint64_t)op[(x >> 4) * 2048 + tc::swz(j, (x >> 1) & 7) + 8 * (x & 1)] << (8 * (j & 7));
        e = F::add(e, typename F::E2{M::mul(in[x], c[0]), M::mul(in[x], c[1])});
    }
    return typename F::E2{F::canon(e.c0), F::canon(e.c1)};
}

// Grid (blocks a slice, slices); clusters of the slices. in: rows of 2^k elements, a multiple of 128 of them; r: the point's
// coordinates from the first of the k variables.
template <class F>
__global__ void __launch_bounds__(DM_BLK, 1)
dot_mma_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, const uint64_t* __restrict__ r, int k, size_t rows) {
    using E2 = typename F::E2;
    using M = pr::MmaField<F>;
    extern __shared__ __align__(1024) uint8_t dm_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dm_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t sm32 = tc::smem_u32(sm);
    constexpr uint32_t cst = DM_STAGES * DM_STAGE;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const int kb = k < DM_SLICE ? k : DM_SLICE;
    E2* share = reinterpret_cast<E2*>(sm + cst + (128u << kb));   // this block's sums of a tile
    E2(*part)[32] = reinterpret_cast<E2(*)[32]>(share);           // first: products over variables 0 .. 4, 5 .. 9, the slice's
    uint64_t* used = reinterpret_cast<uint64_t*>(share + DM_ROWS);   // a stage's MMAs are done
    uint64_t& summed = used[DM_STAGES];                              // a tile's
    uint32_t& tmem_sm = *reinterpret_cast<uint32_t*>(used + DM_STAGES + 1);
    const unsigned slices = gridDim.y, slice = blockIdx.y;
    const size_t tiles = rows / DM_ROWS;
    const int steps = 1 << (kb - 5), count = blockIdx.x < tiles ? (int)((tiles - blockIdx.x + gridDim.x - 1) / gridDim.x) : 0;
    const int total = steps * count;                 // stages of 32 elements of each row
    const auto load = [&](int s) {
        if (s < total) {
            const size_t tile = blockIdx.x + (size_t)(s / steps) * gridDim.x;
            const uint64_t* src = in + ((tile * DM_ROWS) << k) + ((size_t)slice << DM_SLICE) + 32 * (s % steps);
            const uint32_t dst = sm32 + (s % DM_STAGES) * DM_STAGE;
#pragma unroll
            for (int x = 0; x < 8; x++) {
                const uint32_t c = t + x * DM_BLK, row = c >> 4, u = c & 15;
                tc::copy16(dst + (u >> 3) * 16384 + tc::swz(row, u & 7), src + ((size_t)row << k) + 2 * u);
            }
        }
        tc::copy_commit();
    };
    for (int s = 0; s < DM_STAGES - 1; s++) load(s);
    if (t == 0) {
        for (int i = 0; i < DM_STAGES; i++) tc::mbar_init(&used[i], 1);
        tc::mbar_init(&summed, 1);
        tc::mbar_init_fence();
    }
    if (warp == 0) tc::tmem_alloc(&tmem_sm, 32);
    if (t < 96) {
        const int p = t >> 5, first = 5 * p, left = p < 2 ? kb - first : k - DM_SLICE, nb = left < 5 ? left : 5;
        E2 f[5];
#pragma unroll
        for (int b = 0; b < 5; b++) {
            f[b] = E2{1, 0};
            if (b < nb) {
                const E2 x = pr::load2<E2>(r + 2 * (first + b));
                f[b] = ((p < 2 ? lane : (int)slice) >> b) & 1 ? x : F::sub(f[b], x);
            }
        }
        part[p][lane] = F::mul(F::mul(F::mul(f[0], f[1]), F::mul(f[2], f[3])), f[4]);
    }
    __syncthreads();
    if (t < 32) part[1][t] = F::mul(part[1][t], part[2][0]);
    __syncthreads();
    // the operand: by sixteen elements 16 rows (component, byte) of 128 bytes
    for (int x = t; x < (1 << kb); x += DM_BLK) {
        const E2 e = F::mul(part[0][x & 31], part[1][x >> 5]);
#pragma unroll
        for (int comp = 0; comp < 2; comp++) {
            uint64_t f[8], o[8];
            f[0] = comp ? e.c1 : e.c0;
#pragma unroll
            for (int i = 1; i < 8; i++) f[i] = M::red_small(f[i - 1] << 8, (uint32_t)(f[i - 1] >> 56));
            transpose_bytes(f, o);
            uint8_t* p = sm + cst + (x >> 4) * 2048 + 8 * (x & 1);
#pragma unroll
            for (int b = 0; b < 8; b++) *reinterpret_cast<uint64_t*>(p + tc::swz(8 * comp + b, (x >> 1) & 7)) = o[b];
        }
    }
    tc::fence_operands();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_sm;
    bool failed = false;
    tc::Issued issued;   // thread 0's
    for (int s = 0; s < total; s++) {
        const int tile = s / steps, step = s % steps;
        tc::copy_wait<DM_STAGES - 2>();
        tc::fence_operands();
        if (step == 0) tc::fence_before();   // the tile before last has been read out of its columns
        failed = __syncthreads_or(failed);
        if (t == 0 && !failed) {
            tc::fence_after();
            const uint32_t st = sm32 + (s % DM_STAGES) * DM_STAGE;
#pragma unroll
            for (int q = 0; q < 8; q++)
                tc::mma_i8(tmem + 16 * (tile & 1), tc::desc_sw128(st + (q >> 2) * 16384 + (q & 3) * 32, 0),
                           tc::desc_sw128(sm32 + cst + (2 * step + (q >> 2)) * 2048 + (q & 3) * 32, 0), tc::idesc_u8(16, false), step > 0 || q > 0);
            issued.commit_to(tc::smem_u32(&used[s % DM_STAGES]), s / DM_STAGES);
            if (step + 1 == steps) issued.commit_to(tc::smem_u32(&summed), tile);
        }
        // the stage before this one is free for the one after the next
        if (s > 0 && !failed && !tc::mbar_wait(tc::smem_u32(&used[(s - 1) % DM_STAGES]), (uint32_t)(((s - 1) / DM_STAGES) & 1))) failed = true;
        if (!failed) load(s + DM_STAGES - 1);
        if (step + 1 < steps) continue;
        // the tile's sums: a row a thread
        const size_t first = (blockIdx.x + (size_t)tile * gridDim.x) * DM_ROWS;
        if (t < DM_ROWS) {
            if (!failed && !tc::mbar_wait(tc::smem_u32(&summed), (uint32_t)(tile & 1))) failed = true;
            failed = __any_sync(0xffffffffu, failed);
            tc::fence_after();
            uint32_t v[16];
            tc::ld16(tmem + ((uint32_t)(32 * warp) << 16) + 16 * (tile & 1), v);
            E2 e{F::canon(pr::bytes_value_wide<F>(v)), F::canon(pr::bytes_value_wide<F>(v + 8))};
            if (failed) e = plain_row<F>(in + ((first + t) << k) + ((size_t)slice << DM_SLICE), sm + cst, 1 << kb);
            if (slices == 1) pr::store2(out + 2 * (first + t), e.c0, e.c1);
            else share[t] = e;
        }
        if (slices > 1) {
            tc::cluster_sync();
            const uint32_t mine = DM_ROWS / slices;
            if ((uint32_t)t < mine) {
                const uint32_t row = slice * mine + t;
                E2 e{0, 0};
                for (uint32_t q = 0; q < slices; q++) {
                    uint32_t addr;
                    uint64_t c0, c1;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(tc::smem_u32(&share[row])), "r"(q));
                    asm volatile("ld.shared::cluster.v2.u64 {%0, %1}, [%2];" : "=l"(c0), "=l"(c1) : "r"(addr) : "memory");
                    e = F::add(e, E2{c0, c1});
                }
                pr::store2(out + 2 * (first + row), F::canon(e.c0), F::canon(e.c1));
            }
            tc::cluster_sync();
        }
    }
    tc::copy_wait<0>();
    issued.drain();
    tc::fence_before();
    __syncthreads();
    if (warp == 0) tc::tmem_free(tmem, 32);
}

// Variables to bind this way: six and more, at most twelve, of a table of 2^22 elements where a block has its rows to itself (2^21:
// no gain), of 2^24 where a cluster shares them (2^22 elements in rows of 2^10: 41 by rows, 52 here, on 32 blocks). Rows of 2^13 would
// need clusters of eight, which leave a part of each GPC idle (2^24: 72 by rows, 84 here); twelve variables and a short pass for the rest
// are faster than by rows in one: 2^24 elements, m = 13 61 / 50, m = 14 62 / 50, m = 16 (by rows in two passes) 67 / 54; 2^26, m = 14 169 /
// 127. 0: not this way.
inline int dot_mma_vars(int log_n, int m) {
    const int k = m < DM_MAX ? m : DM_MAX;
    return k >= DM_MIN && log_n >= (k < DM_SLICE ? 22 : 24) && log_n - k >= 7 ? k : 0;
}
template <class FOut>
inline int launch_dot_mma(const uint64_t* in, uint64_t* out, const uint64_t* r, int k, size_t rows, cudaStream_t st) {
    using F = typename DotField<FOut>::F;
    const uint32_t smem = dm_smem(k);
    const unsigned slices = k > DM_SLICE ? 1u << (k - DM_SLICE) : 1u;
    // clusters have to fit the SMs of a GPC: a power of two of them, as the tiles are
    unsigned most = (unsigned)sm_count();
    if (slices > 1)
        for (most = 1; 2 * most * slices <= (unsigned)sm_count();) most *= 2;
    const size_t tiles = rows / DM_ROWS;
    if (cudaFuncSetAttribute(dot_mma_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return MB_ERR_CUDA;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(tiles < most ? (unsigned)tiles : most, slices);
    cfg.blockDim = dim3(DM_BLK);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 1; at.val.clusterDim.y = slices; at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    MB_KERNEL_ON("partial_eval_mma", st);
    return cudaLaunchKernelEx(&cfg, dot_mma_kernel<F>, in, out, r, k, rows) == cudaSuccess ? MB_OK : MB_ERR_CUDA;
}

}  // namespace pe
}  // namespace mb
