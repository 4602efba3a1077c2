// Merkle trees over Goldilocks codewords, hashed with Poseidon2 (width 8) or
// Monolith (width 12); the reference picks one at build time (cargo feature
// "monolith", goldilocks-cuda-rs/src/merkle.rs:44-47), here the hash is a
// template policy and both sets of entry points exist side by side.
//
// Tree buffer layout (goldilocks-cuda-rs/src/merkle.rs:266-280): the leaf
// digests, then every layer above them, the root last; 4 words per digest.
// Leaf k hashes the codeword pair k: permute([v0, v1, 0^6])[0..4] for base-field
// pairs, permute([a.c0, a.c1, b.c0, b.c1, 0^4])[0..4] for extension pairs; a node
// is permute(left || right)[0..4] (goldilocks-cuda-rs/src/cpu_poseidon2.rs:145-183,
// device twins goldilocks-cuda-rs/cuda/wrapper.cu:1604-1713). Monolith pads
// the same inputs with zeros to 12 words (goldilocks-cuda-rs/src/cpu_monolith.rs:150-211,
// wrapper.cu:1894-1987). Digests are written canonical.
//
// Large layers are bound by the integer pipes (about 520 modular multiplications for every 32-byte Poseidon2 digest), not
// by HBM: one fully parallel launch per layer, Poseidon2's from P2_TILES_FROM permutations on in tiles of 128
// (poseidon2_tiles.cuh), smaller ones and Monolith's a permutation per thread. The leaves of a folded codeword are hashed by
// the thread that folds them, so a folded codeword is written once and not read back for its tree.
// Small layers are bound by the latency of one permutation: several lanes share a permutation, and a launch covers up to five
// levels (the leaf layer, with its fold, among them). The launches of a tree are a chain (common.cuh): the next one's blocks come up while
// the one before stores its digests (all layers above 2^16 digests, Poseidon2 150 -> 138 us, Monolith 70 -> 61 us; blocks that
// came up any earlier were put where there was room, 179 us).
#pragma once
#include "codeword_fold.cuh"
#include "common.cuh"
#include "gl_poseidon2.cuh"
#include "gl_monolith.cuh"
#include "poseidon2_linear.cuh"
#include "poseidon2_tiles.cuh"

namespace mb {
namespace mk {

constexpr int BLOCK = 128;

// Hash policies. permute(load): the permutation of the state that load(s) writes (it may be asked for again).
// coop(x, l): the permutation spread over LANES lanes, lane l holding word l. COOP_NODES: layers of at most this many
// nodes take the spread form. warp(x, lane, table, ready): a permutation a warp, word lane mod LANES in every copy; ready() is called before the
// table, a Table in shared memory, is used.
struct HashPoseidon2 {
    static constexpr int WIDTH = 8, LANES = 8, MIN_BLOCKS = 6;
    static constexpr size_t COOP_NODES = (size_t)1 << 12;
    static __device__ __forceinline__ uint64_t coop(uint64_t x, int l) { return gl::poseidon2_permute_coop8(x, l); }
    struct Table : P2Warp {
        // in shared memory by asynchronous copies; whole blocks call
        __device__ __forceinline__ void begin() {
            const char* from = reinterpret_cast<const char*>(&g_p2_warp);
            for (unsigned i = 16 * threadIdx.x; i < sizeof(P2Warp); i += 16 * blockDim.x) tc::copy16(tc::smem_u32(this) + i, from + i);
            tc::copy_commit();
        }
        static __device__ __forceinline__ void end() {
            tc::copy_wait<0>();
            __syncthreads();
        }
    };
    template <class Ready>
    static __device__ __forceinline__ uint64_t warp(uint64_t x, int lane, const Table& w, Ready ready) { return poseidon2_permute_warp(x, lane, w, ready); }
    template <class Load>
    static __device__ __forceinline__ void permute(uint64_t* s, Load load) {
        load(s);
        if (!gl::poseidon2_permute_throughput(s)) {
            load(s);
            gl::poseidon2_permute(s);
        }
    }
    static const char* leaves_name() { return "hash_leaves"; }
    static const char* layer_name() { return "compress_layer"; }
};
struct HashMonolith {
    static constexpr int WIDTH = 12, LANES = 16, MIN_BLOCKS = 4;
    static constexpr size_t COOP_NODES = (size_t)1 << 12;
    static __device__ __forceinline__ uint64_t coop(uint64_t x, int l) { return gl::monolith_permute_lanes<false>(x, l); }
    struct Table {
        __device__ __forceinline__ void begin() {}
        static __device__ __forceinline__ void end() { __syncthreads(); }
    };
    template <class Ready>
    static __device__ __forceinline__ uint64_t warp(uint64_t x, int lane, const Table&, Ready) { return gl::monolith_permute_lanes<true>(x, lane); }
    template <class Load>
    static __device__ __forceinline__ void permute(uint64_t* s, Load load) {
        load(s);
        if (!gl::monolith_permute_throughput(s)) {
            load(s);
            gl::monolith_permute(s);
        }
    }
    static const char* leaves_name() { return "monolith_hash_leaves"; }
    static const char* layer_name() { return "monolith_compress_layer"; }
};

__device__ __forceinline__ void store_digest(uint64_t* out, const uint64_t* s) {
    *reinterpret_cast<ulonglong2*>(out) = make_ulonglong2(gl::canon(s[0]), gl::canon(s[1]));
    *reinterpret_cast<ulonglong2*>(out + 2) = make_ulonglong2(gl::canon(s[2]), gl::canon(s[3]));
}

// copies: the digests are written that many times, num_leaves digests apart (a periodic codeword's tree).
template <class H, bool EXT2>
__global__ void __launch_bounds__(BLOCK, H::MIN_BLOCKS)
hash_leaves_kernel(const uint64_t* __restrict__ cw, uint64_t* __restrict__ digests, size_t num_leaves, size_t copies) {
    chain_begin();
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < num_leaves; k += step) {
        uint64_t st[H::WIDTH];
        H::permute(st, [&](uint64_t* s) {
            if (EXT2) {
                ulonglong2 a = *reinterpret_cast<const ulonglong2*>(cw + 4 * k);
                ulonglong2 b = *reinterpret_cast<const ulonglong2*>(cw + 4 * k + 2);
                s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
            } else {
                ulonglong2 a = *reinterpret_cast<const ulonglong2*>(cw + 2 * k);
                s[0] = a.x; s[1] = a.y; s[2] = 0; s[3] = 0;
            }
#pragma unroll
            for (int i = 4; i < H::WIDTH; i++) s[i] = 0;
        });
        if (k + step >= num_leaves) chain_next();
        for (size_t c = 0; c < copies; c++) store_digest(digests + 4 * (c * num_leaves + k), st);
    }
}

// The same for the leaves of a codeword that is folded on the way: leaf k is the pair of elements 2k, 2k + 1 of the folded
// codeword `out` (extension), each from two elements of `in` (MIXED: base field) and one table entry.
struct FoldSource {
    const uint64_t *in, *table;
    uint64_t* out;
    gl::E2 r;
};
template <bool MIXED>
__device__ __forceinline__ gl::E2 folded_element(const FoldSource& f, size_t i, uint64_t r1w) {
    const ulonglong2 e = *reinterpret_cast<const ulonglong2*>(f.table + 2 * i);
    if (MIXED) return bf::fold_pair_base(*reinterpret_cast<const ulonglong2*>(f.in + 2 * i), e, f.r);
    return bf::fold_pair_ext(gl::e2_load(f.in + 4 * i), gl::e2_load(f.in + 4 * i + 2), e, f.r, r1w);
}
template <class H, bool MIXED>
__global__ void __launch_bounds__(BLOCK, H::MIN_BLOCKS)
fold_leaves_kernel(const FoldSource f, uint64_t* __restrict__ digests, size_t num_leaves) {
    chain_begin();
    const size_t step = (size_t)gridDim.x * blockDim.x;
    const uint64_t r1w = gl::mul_small(f.r.c1, 7);
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < num_leaves; k += step) {
        gl::e2_store(f.out + 4 * k, folded_element<MIXED>(f, 2 * k, r1w));
        gl::e2_store(f.out + 4 * k + 2, folded_element<MIXED>(f, 2 * k + 1, r1w));
        uint64_t st[H::WIDTH];
        H::permute(st, [&](uint64_t* s) {   // this thread's own stores
            const gl::E2 a = gl::e2_load(f.out + 4 * k), b = gl::e2_load(f.out + 4 * k + 2);
            s[0] = a.c0; s[1] = a.c1; s[2] = b.c0; s[3] = b.c1;
#pragma unroll
            for (int i = 4; i < H::WIDTH; i++) s[i] = 0;
        });
        if (k + step >= num_leaves) chain_next();
        store_digest(digests + 4 * k, st);
    }
}

// eight words in front of zeros
template <class H>
__device__ __forceinline__ void load_pair(const uint64_t* l, const uint64_t* r, uint64_t* s) {
    const ulonglong2 *p = reinterpret_cast<const ulonglong2*>(l), *q = reinterpret_cast<const ulonglong2*>(r);
    const ulonglong2 a = p[0], b = p[1], c = q[0], d = q[1];
    s[0] = a.x; s[1] = a.y; s[2] = b.x; s[3] = b.y;
    s[4] = c.x; s[5] = c.y; s[6] = d.x; s[7] = d.y;
#pragma unroll
    for (int i = 8; i < H::WIDTH; i++) s[i] = 0;
}
// out[k] = compress(in[2k], in[2k+1]) for k < n, written `copies` times
template <class H>
__global__ void __launch_bounds__(BLOCK, H::MIN_BLOCKS)
compress_layer_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, size_t n, size_t copies) {
    chain_begin();
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
        uint64_t st[H::WIDTH];
        H::permute(st, [&](uint64_t* s) { load_pair<H>(in + 8 * k, in + 8 * k + 4, s); });
        if (k + step >= n) chain_next();
        for (size_t c = 0; c < copies; c++) store_digest(out + 4 * (c * n + k), st);
    }
}

// Left and right children in separate arrays (poseidon2_compress_batch_ffi).
static __global__ void __launch_bounds__(BLOCK)
compress_pairs_kernel(const uint64_t* __restrict__ left, const uint64_t* __restrict__ right,
                      uint64_t* __restrict__ out, size_t n) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
        uint64_t st[8];
        HashPoseidon2::permute(st, [&](uint64_t* s) { load_pair<HashPoseidon2>(left + 4 * k, right + 4 * k, s); });
        store_digest(out + 4 * k, st);
    }
}

// Full Monolith permutation of n width-12 states, canonical outputs.
static __global__ void __launch_bounds__(BLOCK)
monolith_permute_batch_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, size_t n) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
        uint64_t s[12];
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = in[12 * k + i];
        gl::monolith_permute(s);
#pragma unroll
        for (int i = 0; i < 12; i++) out[12 * k + i] = gl::canon(s[i]);
    }
}

// ---- latency-oriented variants: several lanes per permutation ---------------------------
// One layer, eight lanes per permutation (mb_merkle_layer_variant only; the trees use tree_up_coop_kernel): node k is handled by
// eight consecutive threads, each loads a word of the 64-byte input pair and threads 0..3 store the digest.
static __global__ void __launch_bounds__(256)
compress_layer_coop_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, size_t n) {
    const int l = threadIdx.x & 7;
    const size_t groups = ((size_t)gridDim.x * blockDim.x) / 8;
    const size_t rounds = (n + groups - 1) / groups;  // every lane of a warp runs the same trip count
    size_t k = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / 8;
    for (size_t it = 0; it < rounds; it++, k += groups) {
        const bool live = k < n;
        uint64_t x = live ? in[8 * k + l] : 0;
        x = HashPoseidon2::coop(x, l);
        if (live && l < 4) out[4 * k + l] = gl::canon(x);
    }
}

// Up to five layers in one launch: block b hashes `groups` nodes of the lowest layer and the layers above them, `levels`
// layers in all, so that the top one (one node per block) is complete when the grid ends.
//   LEAF_BASE, LEAF_EXT   the lowest layer are the leaves of codeword f.in (base or extension pairs)
//   FOLD_BASE, FOLD_EXT   the same for the codeword that f folds on the way (f.out)
//   NODES                 the lowest layer hashes pairs of the nodes at f.in
// dst: where the lowest layer is stored, size nodes; the layers above follow. With `copies` > 1 every layer is stored that
// many times (a layer then takes copies * size nodes). last_out (may be null; device or pinned host memory) also receives
// the top layer.
// What a small layer costs is one permutation's latency, and issue slots as soon as more than one warp per scheduler
// works on it: a block holds at most 16 permutations, so a layer of 4096 nodes is spread over 256 blocks. A layer with as few nodes in a
// block as warps takes the form with a permutation a warp.
// Blocks are whole warps (the permutations shuffle with the full mask): threads beyond the block's groups compute on zeros
// and store nothing.
enum TreeSource { NODES, LEAF_BASE, LEAF_EXT, FOLD_BASE, FOLD_EXT };
template <class H, TreeSource SRC>
__global__ void __launch_bounds__(256)
tree_up_coop_kernel(const FoldSource f, uint64_t* dst, size_t size, int levels, size_t copies, uint64_t* last_out) {
    __shared__ uint64_t node[16 * 4];
    __shared__ __align__(16) typename H::Table table;
    table.begin();
    chain_begin();
    size_t n = (size_t)1 << (levels - 1);   // this block's nodes of the current layer
    const size_t warps = blockDim.x / 32;
    const auto whole_warps = [](size_t m) { return ((m * H::LANES + 31) & ~(size_t)31) / H::LANES; };
    uint64_t x = 0;
    for (bool lowest = true;; lowest = false) {
        const bool wide = n <= warps;
        const int lanes = wide ? 32 : H::LANES, l = threadIdx.x & (lanes - 1), w = l & (H::LANES - 1);   // w: the lane's word
        const size_t g = threadIdx.x / lanes, k = (size_t)blockIdx.x * n + g;
        const bool live = g < n, in_use = wide ? live : g < whole_warps(n);   // whole warps drop out as the layers shrink
        if (!lowest) {
            x = (live && w < 8) ? node[8 * g + w] : 0;
        } else if (in_use) {
            if (SRC == NODES) {
                x = (live && w < 8) ? f.in[8 * k + w] : 0;
            } else if (SRC == LEAF_BASE) {
                x = (live && w < 2) ? f.in[2 * k + w] : 0;
            } else if (SRC == LEAF_EXT) {
                x = (live && w < 4) ? f.in[4 * k + w] : 0;
            } else {   // one element per lane of the first two, then a word per lane
                gl::E2 e{0, 0};
                if (live && l < 2) {
                    e = folded_element<SRC == FOLD_BASE>(f, 2 * k + l, gl::mul_small(f.r.c1, 7));
                    gl::e2_store(f.out + 2 * (2 * k + l), e);
                }
                const uint64_t c0 = p2_from_lane(e.c0, (threadIdx.x & 31 & ~(lanes - 1)) + ((w >> 1) & 1)),
                               c1 = p2_from_lane(e.c1, (threadIdx.x & 31 & ~(lanes - 1)) + ((w >> 1) & 1));
                x = w < 4 ? (w & 1 ? c1 : c0) : 0;
            }
        }
        if (n == 1) chain_next();
        if (in_use) {
            // all warps are in use in a lowest layer of this form
            x = gl::canon(wide ? H::warp(x, l, table, [&] { if (lowest) H::Table::end(); }) : H::coop(x, l));
        }
        if (live && l < 4) {
            for (size_t c = 0; c < copies; c++) dst[4 * (c * size + k) + l] = x;
        }
        if (n == 1) break;
        if (lowest && !wide) H::Table::end();
        else __syncthreads();            // the pairs of the layer below have been read
        if (live && l < 4) node[4 * g + l] = x;
        __syncthreads();
        dst += 4 * size * copies;
        size /= 2;
        n /= 2;
    }
    if (last_out != nullptr && threadIdx.x < 4) last_out[4 * (size_t)blockIdx.x + threadIdx.x] = x;
}

// Full permutation of n width-8 states (poseidon2_hash_batch_ffi). The compiler's own 80 registers, no spills; held to 64 for eight blocks
// an SM 136 bytes of them go to memory (calls of 1, 2^14 and 2^20 states 27.8, 26.2 and 481 us there, 26.2, 24.8 and 476 here).
static __global__ void __launch_bounds__(BLOCK)
permute_batch_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, size_t n) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += step) {
        uint64_t st[8];
        HashPoseidon2::permute(st, [&](uint64_t* s) { load_pair<HashPoseidon2>(in + 8 * k, in + 8 * k + 4, s); });
        store_digest(out + 8 * k, st);
        store_digest(out + 8 * k + 4, st + 4);
    }
}

// The throughput kernels above for Poseidon2 in tiles of 128 (poseidon2_tiles.cuh): node or leaf k < n of a layer, from f as in
// TreeSource, written `copies` times.
template <TreeSource SRC>
static __global__ void __launch_bounds__(P2_BLK, 1)
poseidon2_tiles_kernel(const FoldSource f, uint64_t* __restrict__ dst, size_t n, size_t copies) {
    extern __shared__ __align__(128) uint8_t p2_sm[];
    __shared__ __align__(8) uint64_t done[P2_TILES];
    __shared__ uint32_t tmem_sm;
    __shared__ int failed;
    const int t = threadIdx.x, g = t / P2_TILE;
    p2_operands(p2_sm);
    chain_begin();
    if (t == 0) {
        failed = 0;
        for (int i = 0; i < P2_TILES; i++) tc::mbar_init(&done[i], 1);
        tc::mbar_init_fence();
    }
    if (t < 32) tc::tmem_alloc(&tmem_sm, 512);
    tc::fence_operands();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    P2Tile tile;
    tile.row = t % P2_TILE;
    tile.tmem = tmem_sm + P2_NA * g + ((tile.row & ~31u) << 16);
    tile.consts = tc::smem_u32(p2_sm);
    tile.rows = p2_sm + P2_ROWS + g * P2_TILE * 16 * P2_UNITS;
    tile.done = tc::smem_u32(&done[g]);
    tile.id = 1 + g;
    tile.failed = &failed;
    const uint64_t r1w = gl::mul_small(f.r.c1, 7);
    // a layer's tiles go to all SMs before a second one to any
    const size_t step = (size_t)gridDim.x * P2_BLK;
    for (size_t k = ((size_t)g * gridDim.x + blockIdx.x) * P2_TILE + tile.row; k - tile.row < n; k += step) {
        const bool live = k < n;
        if ((SRC == FOLD_BASE || SRC == FOLD_EXT) && live) {
            gl::e2_store(f.out + 4 * k, folded_element<SRC == FOLD_BASE>(f, 2 * k, r1w));
            gl::e2_store(f.out + 4 * k + 2, folded_element<SRC == FOLD_BASE>(f, 2 * k + 1, r1w));
        }
        const auto load = [&](uint64_t* s) {
            constexpr int WORDS = SRC == NODES ? 8 : SRC == LEAF_BASE ? 2 : 4;
            const uint64_t* in = (SRC == FOLD_BASE || SRC == FOLD_EXT ? f.out : f.in) + WORDS * k;   // this thread's own stores
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                ulonglong2 v = make_ulonglong2(0, 0);
                if (j < WORDS && live) v = *reinterpret_cast<const ulonglong2*>(in + j);
                s[j] = v.x;
                s[j + 1] = v.y;
            }
        };
        uint64_t s[8];
        load(s);
        if (!p2_permute_tile(tile, s)) {
            load(s);
            gl::poseidon2_permute(s);
        }
        if (live)
            for (size_t c = 0; c < copies; c++) store_digest(dst + 4 * (c * n + k), s);
    }
    chain_next();
    tile.issued.drain();
    tc::fence_before();
    __syncthreads();
    if (t < 32) tc::tmem_free(tmem_sm, 512);
}
// Layers of this many permutations and more go in tiles (us, a thread each and in tiles): 2^15 25.7 and 26.7, 2^16 42.6 and 36.9, 2^17 66 and
// 57, 2^18 123 and 105, 2^19 236 and 192, 2^20 469 and 377. One tile an SM takes 23 us whatever their number (2^13 and 2^14: a thread each 20).
constexpr size_t P2_TILES_FROM = (size_t)1 << 16;
template <TreeSource SRC>
inline void launch_poseidon2_tiles(const FoldSource& f, uint64_t* dst, size_t n, size_t copies, cudaStream_t st) {
    cudaFuncSetAttribute(poseidon2_tiles_kernel<SRC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)P2_SMEM);
    launch_chained(poseidon2_tiles_kernel<SRC>, grid_for(n, P2_TILE, 1), P2_BLK, P2_SMEM, st, f, dst, n, copies);
}
template <class H> constexpr bool in_tiles(size_t) { return false; }
template <> constexpr bool in_tiles<HashPoseidon2>(size_t n) { return n >= P2_TILES_FROM; }

template <class H>
inline void launch_compress_layer(const uint64_t* in, uint64_t* out, size_t n, size_t copies, cudaStream_t st) {
    MB_KERNEL_ON(H::layer_name(), st);
    if (in_tiles<H>(n)) {
        FoldSource f{};
        f.in = in;
        return launch_poseidon2_tiles<NODES>(f, out, n, copies, st);
    }
    launch_chained(compress_layer_kernel<H>, grid_for(n, BLOCK, 16), BLOCK, 0, st, in, out, n, copies);
}

// One launch of tree_up_coop_kernel over a lowest layer of `size` nodes (stored at dst), as many levels as it takes up to
// the layer of `stop` nodes, five at most. Returns the size of the top layer and moves dst to it.
template <class H, TreeSource SRC>
inline size_t launch_tree_up(const FoldSource& f, uint64_t*& dst, size_t size, size_t copies, cudaStream_t st, uint64_t* root_out,
                             size_t stop) {
    int levels = 1;
    while ((size >> levels) >= stop && (size >> levels) >= 1) levels++;
    if (levels > 5 && levels <= 8) levels -= 3;   // the rest have a node a warp throughout
    if (levels > 5) levels = 5;
    const size_t top = size >> (levels - 1);
    // a warp a node up to four nodes a block, LANES lanes above that
    size_t t = (size_t)H::LANES << (levels - 1);
    if (levels <= 3) t = (size_t)32 << (levels - 1);
    else if (t < 128) t = 128;
    {
        MB_KERNEL_ON("tree_up", st);
        launch_chained(tree_up_coop_kernel<H, SRC>, (unsigned)top, (unsigned)t, 0, st, f, dst, size, levels, copies, top == stop ? root_out : nullptr);
    }
    for (; size > top; size /= 2) dst += 4 * size * copies;
    return top;
}

// Every layer above `layer` (`size` nodes, `copies` times) up to the layer of `stop` nodes (1: the root; a power of two
// otherwise, for a caller that hashes the last levels on the host). root_out (may be null; device or pinned host memory)
// receives that last layer: min(size, stop) digests.
template <class H>
inline void finish_layers(uint64_t* layer, size_t size, size_t copies, cudaStream_t st, uint64_t* root_out, size_t stop) {
    if (size <= stop) {
        if (root_out != nullptr) cudaMemcpyAsync(root_out, layer, 32 * size, cudaMemcpyDefault, st);
        return;
    }
    while (size / 2 > H::COOP_NODES && size > stop) {
        launch_compress_layer<H>(layer, layer + 4 * size * copies, size / 2, copies, st);
        layer += 4 * size * copies;
        size /= 2;
    }
    while (size > stop) {
        FoldSource f{};
        f.in = layer;
        uint64_t* dst = layer + 4 * size * copies;
        size = launch_tree_up<H, NODES>(f, dst, size / 2, copies, st, root_out, stop);
        layer = dst;
    }
}

// Layers above the digests already present in tree[0 .. 4*num_leaves).
template <class H>
inline int build_layers(uint64_t* d_tree, size_t num_leaves, cudaStream_t st, uint64_t* root_out = nullptr, size_t stop = 1) {
    finish_layers<H>(d_tree, num_leaves, 1, st, root_out, stop);
    return finish_async();
}

// The leaf layer and everything above it. COOP and THREAD: the kernel forms of the leaf layer.
template <class H, TreeSource COOP, class Thread>
inline int build_from_leaves(const FoldSource& f, uint64_t* d_tree, size_t num_leaves, size_t copies, cudaStream_t st, uint64_t* root_out,
                             size_t stop, Thread thread_form) {
    uint64_t* layer = d_tree;
    size_t size = num_leaves;
    if (num_leaves > H::COOP_NODES) {
        MB_KERNEL_ON(H::leaves_name(), st);
        thread_form();
    } else {
        size = launch_tree_up<H, COOP>(f, layer, num_leaves, copies, st, root_out, num_leaves < stop ? num_leaves : stop);
        if (size <= stop) return finish_async();
    }
    finish_layers<H>(layer, size, copies, st, root_out, stop);
    return finish_async();
}

// stop > 1: the layers above the one of `stop` nodes are left to the caller (finish_layers).
template <class H, bool EXT2>
inline int build_tree(const uint64_t* d_codeword, uint64_t* d_tree, size_t num_leaves, cudaStream_t st,
                      uint64_t* root_out = nullptr, size_t stop = 1) {
    if (!d_codeword || !d_tree || num_leaves < 1 || (num_leaves & (num_leaves - 1))) return MB_ERR_ARG;
    FoldSource f{};
    f.in = d_codeword;
    return build_from_leaves<H, EXT2 ? LEAF_EXT : LEAF_BASE>(f, d_tree, num_leaves, 1, st, root_out, stop, [&] {
        if (in_tiles<H>(num_leaves)) return launch_poseidon2_tiles<EXT2 ? LEAF_EXT : LEAF_BASE>(f, d_tree, num_leaves, 1, st);
        launch_chained(hash_leaves_kernel<H, EXT2>, grid_for(num_leaves, BLOCK, 16), BLOCK, 0, st, d_codeword, d_tree, num_leaves, (size_t)1);
    });
}

// The tree over the codeword that f folds (4 num_leaves elements of f.in, 2 num_leaves of f.out, which is written too).
template <class H, bool MIXED>
inline int fold_tree(const FoldSource& f, uint64_t* d_tree, size_t num_leaves, cudaStream_t st, uint64_t* root_out, size_t stop) {
    return build_from_leaves<H, MIXED ? FOLD_BASE : FOLD_EXT>(f, d_tree, num_leaves, 1, st, root_out, stop, [&] {
        if (in_tiles<H>(num_leaves)) return launch_poseidon2_tiles<MIXED ? FOLD_BASE : FOLD_EXT>(f, d_tree, num_leaves, 1, st);
        launch_chained(fold_leaves_kernel<H, MIXED>, grid_for(num_leaves, BLOCK, 16), BLOCK, 0, st, f, d_tree, num_leaves);
    });
}

// Tree over a base-field codeword that consists of `copies` equal blocks (what
// the foldable-code encoder produces: goldilocks-cuda-rs/cuda/wrapper.cu:1277-1312
// repeats every coefficient 2^log_rate times and its butterflies never mix the
// copies, so after the bit reversal block c equals block 0). Every layer of the
// tree is then periodic too: only the first size/copies nodes of each layer are
// hashed, by kernels that store them `copies` times. The buffer ends up identical to build_tree's.
template <class H>
inline int build_tree_periodic(const uint64_t* d_codeword, uint64_t* d_tree, size_t num_leaves, size_t copies,
                               cudaStream_t st) {
    if (!d_codeword || !d_tree || num_leaves < 1 || (num_leaves & (num_leaves - 1))) return MB_ERR_ARG;
    if (copies < 2 || num_leaves < copies) return build_tree<H, false>(d_codeword, d_tree, num_leaves, st);
    const size_t uniq = num_leaves / copies;
    FoldSource f{};
    f.in = d_codeword;
    int rc = build_from_leaves<H, LEAF_BASE>(f, d_tree, uniq, copies, st, nullptr, 1, [&] {
        if (in_tiles<H>(uniq)) return launch_poseidon2_tiles<LEAF_BASE>(f, d_tree, uniq, copies, st);
        launch_chained(hash_leaves_kernel<H, false>, grid_for(uniq, BLOCK, 16), BLOCK, 0, st, d_codeword, d_tree, uniq, copies);
    });
    if (rc != MB_OK) return rc;
    // one block's root, `copies` times: an ordinary layer
    finish_layers<H>(d_tree + 4 * copies * (2 * uniq - 2), copies, 1, st, nullptr, 1);
    return finish_async();
}

}  // namespace mk
}  // namespace mb
