// tf_candidates_noalloc: the broadphase's candidate pairs for one world of single-shape bodies, computed
// with scratch memory that is part of the library image instead of memory allocated on the device.
//
// The pair rules are the step's (src/world.cpp:788-842 in the reference, k_broadphase here) specialised to
// one shape per body, with shape index = body index: both bodies live, one of them dynamic, one of them
// moving; their bounds overlap after growing one by the sum of both growths; each shape's bounds overlap
// the other body's bounds grown by that sum; and the shapes' bounds, each grown by its own body's growth,
// overlap. The keys (min << 32 | max) come out sorted and unique, as World::Impl::updateContacts leaves them
// (src/world.cpp:868-869). The step's other rules (category/mask filters, jointed pairs, half-space pairs)
// are not applied: the inputs carry no filters, joints or planes.
//
// Scratch: g_pairScratch below, a fixed-size array in the library's device image, its address looked up on every call
// (a context made after a device reset may place the module elsewhere). Nothing here
// allocates device or host memory through CUDA or any other library. Because the scratch is one per device,
// calls whose work overlaps on the device (different streams, or different host threads) race on it and give
// wrong results; issue them on one stream or serialise them.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/twofold_b200.h"
#include "tf_body.cuh"

namespace tfb {

int noteError(int code, const std::string& msg);

namespace {

constexpr int32_t kMaxBodies = TF_NOALLOC_MAX_BODIES;
constexpr int32_t kMaxPairs = TF_NOALLOC_MAX_PAIRS;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;

// Rows (first bodies) and columns (second bodies) of a tile of pair tests: a warp takes kRowsPerWarp rows at once,
// so each second body is loaded once for that many tests, and kTileCols columns, 32 at a time.
constexpr int kRowsPerWarp = 4;
constexpr int kTileWarps = 8;
constexpr int kTileRows = kRowsPerWarp * kTileWarps;
constexpr int kTileCols = 256;
constexpr int kTileWords = kTileCols / 32;
constexpr int kMaxRowTiles = kMaxBodies / kTileRows;
constexpr int kMaxColTiles = kMaxBodies / kTileCols;
constexpr int kMaxWords = kMaxBodies / 32;

// Worlds of at most this many bodies are one CTA's work in one launch. Past it two launches over the device win:
// measured on one B200, 128 bodies take 12.3 us either way, 96 take 10.3 us in one CTA and 11.2 us in two launches,
// 160 take 16.4 us and 12.3 us.
constexpr int kOneCtaBodies = 128;
constexpr int kOneCtaWords = kOneCtaBodies / 32;

struct PairScratch {
    uint32_t hits[(size_t)kMaxBodies * kMaxWords];  // row by row, a bit per second body
    uint32_t tileHits[kMaxRowTiles * kMaxColTiles];  // hits of each tile, row tile by row tile
};

}  // namespace

// 256-byte aligned so that every field above starts on a 16-byte boundary.
static __device__ __align__(256) unsigned char g_pairScratch[sizeof(PairScratch)];

namespace {

__device__ __forceinline__ Vec3 at(const float* p, uint32_t i) { return Vec3{ p[3 * i], p[3 * i + 1], p[3 * i + 2] }; }

struct PairRow {
    Vec3 lo, hi;
    float grow;
    uint32_t flags;
};

__device__ __forceinline__ PairRow pairRow(const float* lo, const float* hi, const float* grow, const uint32_t* flags,
                                           uint32_t i) {
    return PairRow{ at(lo, i), at(hi, i), grow[i], flags[i] };
}

// The pair rules, lower body first.
__device__ __forceinline__ bool pairs(const PairRow& A, const PairRow& B) {
    if (!(A.flags & B.flags & TF_PAIR_LIVE)) { return false; }
    if (!((A.flags | B.flags) & TF_PAIR_DYNAMIC) || !((A.flags | B.flags) & TF_PAIR_MOVING)) { return false; }
    const float gg = A.grow + B.grow;
    const Vec3 reach{ gg, gg, gg };
    if (!boxesOverlap(A.lo - reach, A.hi + reach, B.lo, B.hi)) { return false; }
    if (!boxesOverlap(A.lo, A.hi, B.lo - reach, B.hi + reach)) { return false; }
    if (!boxesOverlap(B.lo, B.hi, A.lo - reach, A.hi + reach)) { return false; }
    const Vec3 g3a{ A.grow, A.grow, A.grow }, g3b{ B.grow, B.grow, B.grow };
    return boxesOverlap(A.lo - g3a, A.hi + g3a, B.lo - g3b, B.hi + g3b);
}

// The hit words of rows row0 .. row0 + kRowsPerWarp of one warp for the 32 second bodies from `first`: lane r gets
// row r's. Bodies past the last one and the diagonal's lower side give no hits.
__device__ __forceinline__ uint32_t hitWords(const PairRow (&rows)[kRowsPerWarp], uint32_t row0, uint32_t first,
                                             uint32_t lane, const float* lo, const float* hi, const float* grow,
                                             const uint32_t* flags, uint32_t n) {
    const uint32_t b = first + lane;
    PairRow B{};
    if (b < n) { B = pairRow(lo, hi, grow, flags, b); }
    uint32_t mine = 0;
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
        const uint32_t word = __ballot_sync(0xffffffffu, b > row0 + r && pairs(rows[r], B));
        if (lane == (uint32_t)r) { mine = word; }
    }
    return mine;
}

__device__ __forceinline__ void loadRows(PairRow (&rows)[kRowsPerWarp], uint32_t row0, const float* lo, const float* hi,
                                         const float* grow, const uint32_t* flags, uint32_t n) {
#pragma unroll
    for (int r = 0; r < kRowsPerWarp; ++r) {
        rows[r] = PairRow{};
        if (row0 + r < n) { rows[r] = pairRow(lo, hi, grow, flags, row0 + r); }
    }
}

// The keys of one row, in order: its words' hits from position `pos` on. Called by a whole warp.
template <class Word>
__device__ __forceinline__ uint32_t emitRow(uint32_t row, uint32_t words, Word word, uint32_t pos, uint32_t lane,
                                            uint64_t* keys, uint32_t capacity) {
    for (uint32_t w0 = row / 32; w0 < words; w0 += 32) {
        uint32_t m = w0 + lane < words ? word(w0 + lane) : 0u;
        const uint32_t c = __popc(m);
        uint32_t x = c;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)lane >= o) { x += y; }
        }
        uint32_t at = pos + x - c;
        while (m) {
            const uint32_t b = (w0 + lane) * 32 + (uint32_t)__ffs(m) - 1;
            m &= m - 1;
            if (at < capacity) { keys[at] = ((uint64_t)row << 32) | b; }
            ++at;
        }
        pos += __shfl_sync(0xffffffffu, x, 31);
    }
    return pos;
}

// Sum over the CTA; every thread calls it, and gets it.
__device__ uint32_t ctaSum(uint32_t v) {
    __shared__ uint32_t s_sum;
    if (threadIdx.x == 0) { s_sum = 0; }
    __syncthreads();
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0 && v) { atomicAdd(&s_sum, v); }
    __syncthreads();
    const uint32_t total = s_sum;
    __syncthreads();
    return total;
}

// Each pair of rows and columns is tested once and each row's columns in ascending order, so the keys need no
// sort and hold no repeats: what is left after the tests is counting where each row's keys start. 4096 bodies of
// 10,195 pairs take 33 us, 1024 take 14 us. (One CTA that appended keys as it found them, then sorted them, took
// 3436 us and 292 us: 147 of 148 SMs idle.)
//
// The tests, a tile of kTileRows x kTileCols pairs a CTA over the tiles that reach above the diagonal: a hit bit
// per pair, and the tile's hits. Bounded by the tests' arithmetic: 4096 bodies are 8.4 million tests.
__global__ void __launch_bounds__(32 * kTileWarps) k_pair_tiles(const float* lo, const float* hi, const float* grow,
                                                                const uint32_t* flags, uint32_t n, PairScratch* S) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t rowTile = blockIdx.y, colTile = blockIdx.x;
    const uint32_t first = colTile * kTileCols, words = (n + 31) / 32;
    uint32_t mine = 0;
    if (first + kTileCols > rowTile * kTileRows) {
        const uint32_t row0 = rowTile * kTileRows + warp * kRowsPerWarp;
        PairRow rows[kRowsPerWarp];
        loadRows(rows, row0, lo, hi, grow, flags, n);
        for (int k = 0; k < kTileWords; ++k) {
            const uint32_t word = first / 32 + k;
            if (word >= words) { break; }
            const uint32_t m = hitWords(rows, row0, first + 32 * k, lane, lo, hi, grow, flags, n);
            if (lane < kRowsPerWarp && row0 + lane < n) { S->hits[(size_t)(row0 + lane) * kMaxWords + word] = m; }
            mine += __popc(m);
        }
    }
    const uint32_t total = ctaSum(mine);
    if (threadIdx.x == 0) { S->tileHits[rowTile * kMaxColTiles + colTile] = total; }
}

// The keys, a row tile a CTA: the tiles before it give where its keys start, its own rows' hits the rest. More
// hits than kMaxPairs leave the keys as they were.
__global__ void __launch_bounds__(32 * kTileWarps) k_pair_keys(uint32_t n, uint64_t* keys, uint32_t capacity, int32_t* count,
                                                               const PairScratch* S) {
    __shared__ uint32_t s_row[kTileRows];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t rowTiles = (n + kTileRows - 1) / kTileRows, colTiles = (n + kTileCols - 1) / kTileCols;
    const uint32_t words = (n + 31) / 32;
    uint32_t before = 0, all = 0;
    for (uint32_t i = tid; i < rowTiles * colTiles; i += blockDim.x) {
        const uint32_t v = S->tileHits[i / colTiles * kMaxColTiles + i % colTiles];
        all += v;
        if (i / colTiles < blockIdx.x) { before += v; }
    }
    all = ctaSum(all);
    before = ctaSum(before);
    if (blockIdx.x == 0 && tid == 0) { *count = all > (uint32_t)kMaxPairs ? -1 : (int32_t)all; }
    if (all > (uint32_t)kMaxPairs) { return; }
    const uint32_t row0 = blockIdx.x * kTileRows;
    for (uint32_t r = warp; r < kTileRows; r += kTileWarps) {
        const uint32_t row = row0 + r;
        uint32_t c = 0;
        if (row < n) {
            for (uint32_t w = row / 32 + lane; w < words; w += 32) { c += __popc(S->hits[(size_t)row * kMaxWords + w]); }
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if (lane == 0) { s_row[r] = c; }
    }
    __syncthreads();
    for (uint32_t r = warp; r < kTileRows && row0 + r < n; r += kTileWarps) {
        const uint32_t pos = before + __reduce_add_sync(0xffffffffu, lane < r ? s_row[lane] : 0u);
        const uint32_t* hits = S->hits + (size_t)(row0 + r) * kMaxWords;
        emitRow(row0 + r, words, [&](uint32_t w) { return hits[w]; }, pos, lane, keys, capacity);
    }
}

// A small world's pairs in one CTA and one launch, the hit bits in shared memory.
__global__ void __launch_bounds__(kThreads) k_pairs_small(const float* lo, const float* hi, const float* grow,
                                                          const uint32_t* flags, uint32_t n, uint64_t* keys,
                                                          uint32_t capacity, int32_t* count) {
    __shared__ uint32_t s_hits[kOneCtaBodies * kOneCtaWords];
    __shared__ uint32_t s_row[kOneCtaBodies];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, words = (n + 31) / 32;
    for (uint32_t row0 = warp * kRowsPerWarp; row0 < n; row0 += kWarps * kRowsPerWarp) {
        PairRow rows[kRowsPerWarp];
        loadRows(rows, row0, lo, hi, grow, flags, n);
        uint32_t c = 0;
        for (uint32_t w = row0 / 32; w < words; ++w) {
            const uint32_t m = hitWords(rows, row0, 32 * w, lane, lo, hi, grow, flags, n);
            if (lane < kRowsPerWarp && row0 + lane < n) { s_hits[(row0 + lane) * kOneCtaWords + w] = m; }
            c += __popc(m);
        }
        if (lane < kRowsPerWarp && row0 + lane < n) { s_row[row0 + lane] = c; }
    }
    __syncthreads();
    uint32_t all = 0;
    for (uint32_t r = lane; r < n; r += 32) { all += s_row[r]; }
    all = __reduce_add_sync(0xffffffffu, all);
    if (tid == 0) { *count = all > (uint32_t)kMaxPairs ? -1 : (int32_t)all; }
    if (all > (uint32_t)kMaxPairs) { return; }
    for (uint32_t row = warp; row < n; row += kWarps) {
        uint32_t before = 0;
        for (uint32_t r = lane; r < row; r += 32) { before += s_row[r]; }
        before = __reduce_add_sync(0xffffffffu, before);
        emitRow(row, words, [&](uint32_t w) { return s_hits[row * kOneCtaWords + w]; }, before, lane, keys, capacity);
    }
}

// The scratch's device address in the current context, looked up on every call (a host-side table lookup of the
// loaded module, cheap): a context made after a device reset may place the module elsewhere.
int scratchAddress(PairScratch** out) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_pairScratch);
    if (e != cudaSuccess) {
        return noteError(TF_E_CUDA, std::string("tf_candidates_noalloc: cudaGetSymbolAddress: ") + cudaGetErrorString(e));
    }
    *out = static_cast<PairScratch*>(p);
    return TF_OK;
}

}  // namespace
}  // namespace tfb

extern "C" {

TF_API int tf_candidates_noalloc(const float* lo, const float* hi, const float* grow, const uint32_t* flags, int32_t n,
                                 uint64_t* keys, int32_t capacity, int32_t* count, void* stream) {
    using namespace tfb;
    if (n < 0 || capacity < 0) { return noteError(TF_E_INVALID, "tf_candidates_noalloc: negative size"); }
    if (n > kMaxBodies) {
        return noteError(TF_E_CAPACITY, "tf_candidates_noalloc: " + std::to_string(n) + " bodies; at most " +
                                            std::to_string(kMaxBodies) + " fit its fixed scratch");
    }
    if (!count || (n > 0 && (!lo || !hi || !grow || !flags)) || (capacity > 0 && !keys)) {
        return noteError(TF_E_INVALID, "tf_candidates_noalloc: null pointer");
    }
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (n <= kOneCtaBodies) {
        k_pairs_small<<<1, kThreads, 0, st>>>(lo, hi, grow, flags, (uint32_t)n, keys, (uint32_t)capacity, count);
    } else {
        PairScratch* S = nullptr;
        const int rc = scratchAddress(&S);
        if (rc != TF_OK) { return rc; }
        const unsigned rowTiles = (unsigned)(n + kTileRows - 1) / kTileRows, colTiles = (unsigned)(n + kTileCols - 1) / kTileCols;
        k_pair_tiles<<<dim3(colTiles, rowTiles), 32 * kTileWarps, 0, st>>>(lo, hi, grow, flags, (uint32_t)n, S);
        k_pair_keys<<<rowTiles, 32 * kTileWarps, 0, st>>>((uint32_t)n, keys, (uint32_t)capacity, count, S);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) { return noteError(TF_E_CUDA, std::string("tf_candidates_noalloc: launch: ") + cudaGetErrorString(e)); }
    return TF_OK;
}

}  // extern "C"
