// pbf_bins.cu -- the step's reorder by cell, and the grid build on caller-owned
// memory: a stable counting sort.
//
// A rebuild orders the particles by cell key, equal keys in their previous
// order (src/pbf/spatial_grid.cu:188-204, a stable radix sort and the cell
// ranges).  The keys are cell numbers, and the cell table first[] (the exclusive
// scan of the cells' counts) is wanted in any case, so a counting sort needs
// no digit passes:
//   the kernel that computes a key also counts it (atomicAdd on the cell; the
//   returned place is this particle's arrival among the cell's particles,
//   any order);
//   k_bin_scan          counts -> first[];
//   k_bin_scatter       particle numbers into their cell's slots, in arrival
//                       order (k_bin_small: both in one launch);
//   k_bin_gather        per slot, the particle's place among its cell's ones in
//                       their previous order (how many of the cell's numbers
//                       are smaller), and the reorder to that place.  The
//                       result is the stable sort's whatever the arrivals.
// The last step reads a cell's m numbers m times; the walk that follows tests
// at least as many pairs of each cell, so no distribution of the particles
// makes it the larger cost.
//
// Bound by the latency of its dependent loads (2 launches a rebuild up to 8,192
// cells, 3 above, and one more where the scan's tile sums are not counted with
// the keys) against the radix sort's 4 to 9 launches and the gather's search of
// first[].  Measured on a GB300, radix sort and gather against this, five
// rebuilds of a frame: 81 -> 64 us at 1,024 particles, 137 -> 85 at 65,536,
// 387 -> 215 at 262,144 (two substeps), 310 -> 196 at 1,048,576, 1.67 -> 1.07
// ms at 8,388,608.
#include "pbf_kernels.cuh"

#include <algorithm>

namespace pbf {

namespace {

__device__ __forceinline__ bool fatal(const unsigned* status) {
    return status != nullptr && (__ldcg(status) & kStatusFatalMask) != 0u;
}

// Exclusive scan over the block's values (one per thread); total: their sum.
template <int THREADS>
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* warp_sums, uint32_t& total) {
    constexpr int kWarps = THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    uint32_t w = lane < kWarps ? warp_sums[lane] : 0u;  // every warp scans the warps' sums
#pragma unroll
    for (int o = 1; o < kWarps; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
    }
    total = __shfl_sync(0xffffffffu, w, kWarps - 1);
    const uint32_t before = __shfl_sync(0xffffffffu, w, max(warp - 1, 0));
    return (warp ? before : 0u) + incl - v;
}

// Cells per thread in the scans: few where the launch is short and its blocks
// should be many, 8 for large tables.
constexpr int kFew = 2, kMany = 8;

// ITEMS consecutive counts of the thread (0 past the last cell).  PADDED: the
// array is 16-byte aligned and padded to a multiple of kMany cells
// (bin_count_words); else a caller's array of `cells` words.
template <int ITEMS, bool PADDED = true>
__device__ __forceinline__ uint32_t load_counts(const uint32_t* __restrict__ count, uint32_t at,
                                                uint32_t cells, uint32_t (&v)[ITEMS]) {
    uint32_t sum = 0u;
    if constexpr (PADDED) {
#pragma unroll
        for (int q = 0; q < ITEMS; q += 2) {
            const uint2 w = at + q < cells ? __ldcg(reinterpret_cast<const uint2*>(count + at + q))
                                           : make_uint2(0u, 0u);
            v[q] = w.x;
            v[q + 1] = w.y;
            sum += w.x + w.y;
        }
    } else {
#pragma unroll
        for (int q = 0; q < ITEMS; ++q) {
            v[q] = at + q < cells ? __ldcg(&count[at + q]) : 0u;
            sum += v[q];
        }
    }
    return sum;
}

// Up to kSmallCells cells: every block scans all counts into shared memory
// (32 KB at most, from L2) and places its particles; block 0 writes first[].
constexpr int kSmallThreads = 1024;
constexpr int kItems = kMany;
constexpr uint32_t kSmallCells = kSmallThreads * kItems;
__global__ void __launch_bounds__(kSmallThreads)
k_bin_small(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ place,
            const uint32_t* __restrict__ count, int n, uint32_t cells, int* __restrict__ first,
            uint32_t* __restrict__ list, const unsigned* __restrict__ status) {
    __shared__ uint32_t start[kSmallCells];
    __shared__ uint32_t warp_sums[kSmallThreads / 32];
    const int i = blockIdx.x * kSmallThreads + threadIdx.x;
    const uint32_t key = i < n ? keys[i] : 0u, at = i < n ? place[i] : 0u;
    uint32_t v[kItems], total;
    const uint32_t c0 = threadIdx.x * kItems;
    const uint32_t sum = load_counts<kItems>(count, c0, cells, v);
    if (__syncthreads_or(fatal(status))) return;
    uint32_t run = block_scan<kSmallThreads>(sum, warp_sums, total);
#pragma unroll
    for (int q = 0; q < kItems; ++q) {
        start[c0 + q] = run;
        if (blockIdx.x == 0 && c0 + q <= cells) first[c0 + q] = static_cast<int>(run);
        run += v[q];
    }
    if (blockIdx.x == 0 && cells == kSmallCells && threadIdx.x == 0)
        first[cells] = static_cast<int>(total);
    __syncthreads();
    const uint32_t slot = start[key] + at;
    if (i < n && slot < static_cast<uint32_t>(n)) list[slot] = static_cast<uint32_t>(i);
}

constexpr int kScanThreads = 512;
// A scan block's tile of counts: kFew cells a thread up to kFewCells (32,768
// cells: 8.4 -> 5.4 us), kMany above.  The tiles' sums are counted with the keys
// (put_key), a warp's particles of a tile at once, where the particles are in the
// last rebuild's order and at most kTileCountMax: frame at 65,536 particles 244 ->
// 238 us, pass at 262,144 (two substeps) 2,174 -> 2,150.  At 8,388,608 the atomics
// cost more than they save (13.6 -> 14.2 ms), at 1,048,576 still a little less
// (four frames 7,589 -> 7,542 us); the line was drawn above the two sizes timed at
// first.  With particles in any order neighbouring threads share no tile
// (200,003 positions 31 -> 70 us).  Else
// k_bin_sums reads the counts (5.0 us at 1,048,576 particles) or, up to
// kDirectCells, every scan block those before its own tile (at 32,768 cells 5.4 us
// against 3.8 + 5.9).
constexpr uint32_t kDirectCells = 32768;
constexpr size_t kTileCountMax = size_t(1) << 19;
constexpr uint32_t kFewCells = 1u << 20;
int tile_shift(uint64_t cells) {
    constexpr int few = 10, many = 12;
    static_assert(kScanThreads * kFew == 1 << few && kScanThreads * kMany == 1 << many, "");
    return cells <= kFewCells ? few : many;
}
size_t tile_count(uint64_t cells) {
    return static_cast<size_t>((cells + (uint64_t(1) << tile_shift(cells)) - 1) >>
                               tile_shift(cells));
}

template <int ITEMS, bool PADDED = true>
__global__ void __launch_bounds__(kScanThreads)
k_bin_sums(const uint32_t* __restrict__ count, uint32_t cells, uint32_t* __restrict__ sums,
           const unsigned* __restrict__ status) {
    __shared__ uint32_t warp_sums[kScanThreads / 32];
    if (__syncthreads_or(fatal(status))) return;
    uint32_t v[ITEMS], total;
    block_scan<kScanThreads>(
        load_counts<ITEMS, PADDED>(count, (blockIdx.x * kScanThreads + threadIdx.x) * ITEMS,
                                   cells, v),
        warp_sums, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

// sums: the tiles' sums, or null (every block sums the counts before its tile).
template <int ITEMS>
__global__ void __launch_bounds__(kScanThreads)
k_bin_scan(const uint32_t* __restrict__ count, uint32_t cells, const uint32_t* __restrict__ sums,
           int* __restrict__ first, const unsigned* __restrict__ status) {
    __shared__ uint32_t warp_sums[2][kScanThreads / 32];
    uint32_t v[ITEMS], base, total;
    const uint32_t c0 = (blockIdx.x * kScanThreads + threadIdx.x) * ITEMS;
    const uint32_t sum = load_counts<ITEMS>(count, c0, cells, v);
    uint32_t before = 0u;
    if (sums) {
        for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kScanThreads) before += sums[t];
    } else {
        const uint4* c4 = reinterpret_cast<const uint4*>(count);
        const uint32_t end = blockIdx.x * (kScanThreads * ITEMS / 4);
#pragma unroll 8
        for (uint32_t t = threadIdx.x; t < end; t += kScanThreads) {
            const uint4 w = __ldcg(&c4[t]);
            before += w.x + w.y + w.z + w.w;
        }
    }
    if (__syncthreads_or(fatal(status))) return;
    block_scan<kScanThreads>(before, warp_sums[0], base);
    uint32_t run = base + block_scan<kScanThreads>(sum, warp_sums[1], total);
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        if (c0 + q <= cells) first[c0 + q] = static_cast<int>(run);
        run += v[q];
    }
    if (c0 + ITEMS == cells) first[cells] = static_cast<int>(run);
}

__global__ void __launch_bounds__(kBlock)
k_bin_scatter(const uint32_t* __restrict__ keys, const uint32_t* __restrict__ place,
              const int* __restrict__ first, int n, uint32_t* __restrict__ list,
              const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    const uint32_t slot = static_cast<uint32_t>(__ldg(&first[keys[i]])) + place[i];
    if (slot < static_cast<uint32_t>(n)) list[slot] = static_cast<uint32_t>(i);
}

// Thread s < n reorders the particle in slot s; thread s < cells clears the
// count of cell s (s < tiles: the sum of tile s) for the next rebuild.  FINAL: with the velocity update of
// k_finalize for the same particle (as a launch of its own it adds 2 us to a
// frame of up to 65,536 particles, 11 to one of 1,048,576).
template <bool FINAL>
__global__ void __launch_bounds__(kBlock)
k_bin_gather(const uint32_t* __restrict__ list, const uint32_t* __restrict__ keys,
             const int* __restrict__ first, uint32_t* __restrict__ count, uint32_t cells,
             uint32_t* __restrict__ sums, uint32_t tiles, const float4* __restrict__ xs_in, float4* __restrict__ xs_out,
             const uint32_t* __restrict__ org_in, uint32_t* __restrict__ org_out,
             uint32_t* __restrict__ perm, float* __restrict__ sx, float* __restrict__ sy,
             float* __restrict__ sz, int n, FinalUpdate f, const unsigned* __restrict__ status) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (fatal(status)) return;
    if (static_cast<uint32_t>(s) < cells) count[s] = 0u;
    if (static_cast<uint32_t>(s) < tiles) sums[s] = 0u;
    if (s >= n) return;
    const uint32_t p = list[s];
    const uint32_t key = keys[p];
    const float4 q = xs_in[p];
    const uint32_t o = org_in ? org_in[p] : p;
    const int a = __ldg(&first[key]), b = __ldg(&first[key + 1u]);
    float4 v{}, vin{};
    uint32_t id = 0u;
    if constexpr (FINAL) {
        v = updated_velocity(f.x_old[o], q, f.v_old[o].w, f.inv_dt);
        vin = f.vin_old[o];
        id = f.id_old[o];
    }
    int dst = a;
    for (int k = a; k < b; ++k) dst += __ldg(&list[k]) < p ? 1 : 0;
    if constexpr (FINAL) {
        f.v_new[dst] = v;
        f.vin_new[dst] = vin;
        f.id_new[dst] = id;
    }
    xs_out[dst] = q;
    sx[dst] = q.x;
    sy[dst] = q.y;
    sz[dst] = q.z;
    org_out[dst] = o;
    if (perm) perm[dst] = p;
}

// --- the grid build alone (launch_bin_grid) ----------------------------------
// Bound by its launches and their dependent loads: 200,003 positions in 184,320
// cells 60 us by the radix sort, 31 here (floor of its bytes about 1 us).
// The caller's cell_start holds the counts until the scan writes the ranges in
// place.  Equal keys may be many (no walk follows that would cost more than
// their ranks): cells of more than kBigCell positions are ranked through a bit
// per position, in units of up to kUnit of them.
constexpr uint32_t kBigCell = 256, kUnit = 8192;
constexpr int kGridMax = 262144;        // positions
constexpr int kBitWords = kGridMax / 32;
constexpr uint32_t kMaxParts = 32;
constexpr uint32_t kUnits = kGridMax / kBigCell + kGridMax / kUnit + 3 * kMaxParts;  // at most
constexpr uint32_t kCellBits = 27, kCellMask = (1u << kCellBits) - 1u;  // of a unit's entry
static_assert(8ull * kGridMax + 65536 <= kCellMask && kMaxParts <= 1u << (32 - kCellBits),
              "a unit's cell and number fit a word");
constexpr unsigned kBigBlocks = 4 * 152;

// Units of a cell of m positions: one for kUnit of them, kMaxParts above 8.
__device__ __forceinline__ uint32_t parts_of(uint32_t m) {
    const uint32_t parts = (m + kUnit - 1u) / kUnit;
    return parts <= 8u ? parts : kMaxParts;
}

__global__ void __launch_bounds__(kBlock)
k_grid_count(const float4* __restrict__ pos, int n, GridConst g, uint32_t* __restrict__ keys,
             uint32_t* __restrict__ place, uint32_t* __restrict__ count,
             uint32_t* __restrict__ units) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *units = 0u;  // for k_grid_scan
    // One atomic per warp and cell: all positions may be in one.
    const uint32_t key = i < n ? key_of(g, pos[i]) : 0xffffffffu;  // past any cell
    const unsigned same = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    uint32_t at = 0u;
    if (i < n && lane == leader) at = atomicAdd(&count[key], static_cast<uint32_t>(__popc(same)));
    at = __shfl_sync(0xffffffffu, at, leader);
    if (i >= n) return;
    keys[i] = key;
    place[i] = at + static_cast<uint32_t>(__popc(same & ((1u << lane) - 1u)));
}

// Counts into ranges, -1 for empty cells; the units of the big cells into
// units[1..], their number into units[0].  A block reads no counts but its own
// tile's, so that the starts can take their place.
template <int ITEMS>
__global__ void __launch_bounds__(kScanThreads)
k_grid_scan(uint32_t* count_start, uint32_t cells, const uint32_t* __restrict__ sums,
            int* __restrict__ cell_end, uint32_t* __restrict__ units) {
    __shared__ uint32_t warp_sums[2][kScanThreads / 32];
    uint32_t v[ITEMS], base, total, before = 0u;
    const uint32_t c0 = (blockIdx.x * kScanThreads + threadIdx.x) * ITEMS;
    const uint32_t sum = load_counts<ITEMS, false>(count_start, c0, cells, v);
    for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kScanThreads) before += sums[t];
    block_scan<kScanThreads>(before, warp_sums[0], base);
    uint32_t run = base + block_scan<kScanThreads>(sum, warp_sums[1], total);
#pragma unroll
    for (int q = 0; q < ITEMS; ++q) {
        if (c0 + q >= cells) break;
        count_start[c0 + q] = v[q] ? run : 0xffffffffu;
        run += v[q];
        cell_end[c0 + q] = v[q] ? static_cast<int>(run) : -1;
        if (v[q] > kBigCell) {
            const uint32_t parts = parts_of(v[q]), u = atomicAdd(units, parts);
            for (uint32_t j = 0; j < parts; ++j) units[1 + u + j] = c0 + q | j << kCellBits;
        }
    }
}

// Thread s of the first blocks places the position in slot s among its cell's,
// in index order.  The last kBigBlocks take the units of the big cells: part j
// numbers the cell's positions in the j-th of equal ranges of indices by their
// bits, after the cell's positions before that range.  It reads the cell's list,
// or, where that is a quarter of all or more, the keys up to the range's end:
// 262,144 positions in one of 262,144 cells 85 us by the list, 63 by the keys;
// 13 cells of 20,000 46 and 120 (radix sort 60 in both).  keys: 16-byte aligned.
__global__ void __launch_bounds__(kBlock)
k_grid_rank(const uint32_t* __restrict__ list, const uint32_t* __restrict__ keys,
            const int* __restrict__ start, const int* __restrict__ end, int n,
            const uint32_t* __restrict__ units, uint32_t* __restrict__ sorted_keys,
            uint32_t* __restrict__ sorted_idx) {
    constexpr int kAhead = 8;  // loads in flight
    __shared__ uint32_t bits[kBitWords + kBlock];
    __shared__ uint32_t warp_sums[2][kBlock / 32];
    const unsigned rank_blocks = gridDim.x - kBigBlocks;
    if (blockIdx.x < rank_blocks) {
        const int s = blockIdx.x * kBlock + threadIdx.x;
        if (s >= n) return;
        const uint32_t p = list[s], key = keys[p];
        sorted_keys[s] = key;  // slots are in cell order
        const int a = __ldg(&start[key]), b = __ldg(&end[key]);
        if (b - a > static_cast<int>(kBigCell)) return;
        int dst = a;
        for (int k = a; k < b; ++k) dst += __ldg(&list[k]) < p ? 1 : 0;
        sorted_idx[dst] = p;
        return;
    }
    const uint32_t todo = units[0];
    for (uint32_t u = blockIdx.x - rank_blocks; u < todo; u += kBigBlocks) {
        const uint32_t unit = units[1 + u], cell = unit & kCellMask, j = unit >> kCellBits;
        const int a = __ldg(&start[cell]), b = __ldg(&end[cell]);
        const uint32_t parts = parts_of(static_cast<uint32_t>(b - a));
        const uint32_t words = (static_cast<uint32_t>(n) + 31u) / 32u;
        const uint32_t w0 = words * j / parts, w1 = words * (j + 1u) / parts;
        // A thread's words: 2^sh side by side and one of padding (bank conflicts).
        int sh = 0;
        while (w1 - w0 > static_cast<uint32_t>(kBlock << sh)) ++sh;
        for (int w = threadIdx.x; w < (kBlock << sh) + kBlock; w += kBlock) bits[w] = 0u;
        __syncthreads();
        uint32_t before = 0u;
        if (parts < kMaxParts) {
            for (int k = a + static_cast<int>(threadIdx.x); k < b; k += kAhead * kBlock) {
                uint32_t p[kAhead];
#pragma unroll
                for (int q = 0; q < kAhead; ++q)
                    p[q] = k + q * kBlock < b ? __ldg(&list[k + q * kBlock]) : 0xffffffffu;
#pragma unroll
                for (int q = 0; q < kAhead; ++q) {
                    const uint32_t w = p[q] >> 5, at = w - w0;
                    before += w < w0 ? 1u : 0u;
                    if (at < w1 - w0) atomicOr(&bits[at + (at >> sh)], 1u << (p[q] & 31u));
                }
            }
        } else {
            const uint4* keys4 = reinterpret_cast<const uint4*>(keys);
#pragma unroll 8
            for (uint32_t k = threadIdx.x; k < 8u * w0; k += kBlock) {
                const uint4 q = __ldg(&keys4[k]);
                before += (q.x == cell) + (q.y == cell) + (q.z == cell) + (q.w == cell);
            }
            const uint32_t lane = threadIdx.x & 31u;
#pragma unroll 4
            for (uint32_t w = w0 + (threadIdx.x >> 5); w < w1; w += kBlock / 32) {
                const uint32_t i = 32u * w + lane;
                const uint32_t key = i < static_cast<uint32_t>(n) ? __ldg(&keys[i]) : 0xffffffffu;
                const unsigned in = __ballot_sync(0xffffffffu, key == cell);
                if (lane == 0u) bits[(w - w0) + ((w - w0) >> sh)] = in;
            }
        }
        __syncthreads();
        const uint32_t* mine = &bits[(threadIdx.x << sh) + threadIdx.x];
        uint32_t set = 0u, total, below;
        for (int w = 0; w < 1 << sh; ++w) set += __popc(mine[w]);
        block_scan<kBlock>(before, warp_sums[0], below);
        int dst = a + static_cast<int>(below + block_scan<kBlock>(set, warp_sums[1], total));
        for (int w = 0; w < 1 << sh; ++w) {
            const uint32_t i0 = 32u * (w0 + (threadIdx.x << sh) + w);
            for (uint32_t m = mine[w]; m; m &= m - 1u)
                sorted_idx[dst++] = i0 + static_cast<uint32_t>(__ffs(m) - 1);
        }
        __syncthreads();
    }
}

}  // namespace

bool bins_apply(size_t n, uint64_t cells) {
    return cells <= std::min<uint64_t>(8 * uint64_t(n) + 65536, uint64_t(1) << 30);
}

size_t bin_count_words(uint64_t cells) {
    return static_cast<size_t>((cells + kMany - 1) / kMany * kMany) + tile_count(cells);
}

// Above kSmallCells cells the words after the counts hold the tiles' sums.
static uint32_t* sums_of(const CellBins& b, uint64_t cells) {
    return b.count + (cells + kMany - 1) / kMany * kMany;
}

CellBins make_bins(uint32_t* count, uint32_t* place, uint64_t cells, size_t n) {
    CellBins b;
    b.count = count;
    b.place = place;
    if (cells > kSmallCells && n <= kTileCountMax) {
        b.sums = sums_of(b, cells);
        b.shift = tile_shift(cells);
    }
    return b;
}

void launch_bin_order(const CellBins& b, const uint32_t* keys, int* first, uint32_t* list, int n,
                      uint64_t cells, const unsigned* status, cudaStream_t st) {
    const uint32_t nc = static_cast<uint32_t>(cells);
    if (nc <= kSmallCells) {
        launch_k(k_bin_small, blocks_for(n, kSmallThreads), kSmallThreads, st, keys, b.place,
                 b.count, n, nc, first, list, status);
        return;
    }
    const bool few = nc <= kFewCells;
    const unsigned tiles = static_cast<unsigned>(tile_count(cells));
    uint32_t* sums = b.sums;
    if (!sums && nc > kDirectCells) {
        sums = sums_of(b, cells);
        launch_k(few ? k_bin_sums<kFew> : k_bin_sums<kMany>, tiles, kScanThreads, st, b.count, nc,
                 sums, status);
    }
    launch_k(few ? k_bin_scan<kFew> : k_bin_scan<kMany>, tiles, kScanThreads, st, b.count, nc,
             sums, first, status);
    launch_k(k_bin_scatter, blocks_for(n), kBlock, st, keys, b.place, first, n, list, status);
}

void launch_bin_gather(const CellBins& b, const uint32_t* list, const uint32_t* keys,
                       const int* first, uint64_t cells, const float4* xs_in, float4* xs_out,
                       const uint32_t* org_in, uint32_t* org_out, uint32_t* perm, float* sx,
                       float* sy, float* sz, int n, const unsigned* status, cudaStream_t st,
                       const FinalUpdate* final_update) {
    const uint64_t threads = std::max<uint64_t>(static_cast<uint64_t>(n), cells);
    launch_k(final_update ? k_bin_gather<true> : k_bin_gather<false>, blocks_for(threads), kBlock, st, list, keys, first, b.count,
             static_cast<uint32_t>(cells), b.sums,
             b.sums ? static_cast<uint32_t>(tile_count(cells)) : 0u, xs_in, xs_out, org_in, org_out, perm, sx, sy, sz, n,
             final_update ? *final_update : FinalUpdate{}, status);
}

size_t bin_grid_words(uint64_t cells) {
    return tile_count(cells) + 1 + kUnits;
}

void launch_bin_grid(const float4* pos, int n, const GridConst& g, uint64_t cells,
                     uint32_t* sorted_keys, uint32_t* sorted_idx, int* cell_start, int* cell_end,
                     uint32_t* keys, uint32_t* place, uint32_t* list, uint32_t* scratch,
                     cudaStream_t st) {
    const uint32_t nc = static_cast<uint32_t>(cells);
    const bool few = nc <= kFewCells;
    const unsigned tiles = static_cast<unsigned>(tile_count(cells));
    uint32_t* count = reinterpret_cast<uint32_t*>(cell_start);
    uint32_t *sums = scratch, *units = scratch + tiles;
    launch_error_check(cudaMemsetAsync(count, 0, cells * sizeof(uint32_t), st));
    launch_k(k_grid_count, blocks_for(n), kBlock, st, pos, n, g, keys, place, count, units);
    if (tiles > 1)
        launch_k(few ? k_bin_sums<kFew, false> : k_bin_sums<kMany, false>, tiles, kScanThreads, st,
                 count, nc, sums, nullptr);
    launch_k(few ? k_grid_scan<kFew> : k_grid_scan<kMany>, tiles, kScanThreads, st, count, nc,
             sums, cell_end, units);
    launch_k(k_bin_scatter, blocks_for(n), kBlock, st, keys, place, cell_start, n, list, nullptr);
    launch_k(k_grid_rank, blocks_for(n) + kBigBlocks, kBlock, st, list, keys, cell_start, cell_end,
             n, units, sorted_keys, sorted_idx);
}

}  // namespace pbf
