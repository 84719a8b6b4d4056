// pbf_kernels.cu -- per-particle kernels of the PBF step for sm_103a.
//
// Hot path per constraint iteration (reference: src/pbf/pbf_solver.cu:210-258):
//   k_predict        integrate + v_in copy + first cell keys      (integration.cu:6-32)
//   [rebuild]        stable counting sort by cell: first[] (lower bound of
//                    every cell key; the row walk's form of cellStart/cellEnd),
//                    reorder of the predicted positions, composed permutation
//                    (pbf_bins.cu; spatial_grid.cu:123-196).  With far more
//                    cells than particles a radix sort (pbf_sort.cu) and
//                    k_gather_first.
//   k_search<true>   neighbour walk + lambda in one pass           (neighbors.cu:3-91,
//                                                                  pbf_solver_kernels.cu:26-105)
//   k_delta_apply    delta p + apply + collision projection + next keys
//                                                                 (pbf_solver_kernels.cu:108-193,
//                                                                  collision_system.cu:133-172)
// After the last iteration (pbf_solver.cu:260-323), after the final rebuild:
//   k_finalize       gather x, v_in, ids by the composite permutation + velocity update
//                    (part of the final rebuild's reorder in pbf_bins.cu)
//   k_search_xsph    rebuilt lists for the velocity terms + XSPH over them
//                    (k_search<false> when XSPH is off)
//   k_vorticity, k_confine   (pbf_solver_kernels.cu:268-385), collision velocity
//                    response fused into the last velocity kernel
//   k_xsph           XSPH alone (stage API)
//
// Every floating-point operation uses the explicit-rounding helpers of
// pbf_math.cuh so the host oracle reproduces the step bit for bit.
#include "pbf_kernels.cuh"

#include "pbf_common.h"
#include "pbf_device.cuh"

#include <algorithm>

namespace pbf {

void launch_error_check(cudaError_t e) { cuda_check(e); }

// Register cap of a neighbour-loop kernel bound by the latency of its
// dependent gathers (list index, then the neighbour's data): fewer registers
// a thread, more warps in flight (k_delta_apply: 58 -> 48 registers, 6 % faster
// at 1M particles; no spills with the exponents 1 to 4, 4 bytes batched, 16 to 20
// with the exponent read at run time).
#define PBF_GATHER_REGS(r) __maxnreg__(r)


namespace {

// ---------------------------------------------------------------------------
// integrate + collision input velocity + keys of the first rebuild
// ---------------------------------------------------------------------------
template <bool B>
__global__ void __launch_bounds__(kBlock)
k_predict(const float4* __restrict__ x, const float4* __restrict__ v, float4* __restrict__ xs,
          float4* __restrict__ vin, uint32_t* __restrict__ keys, CellBins bins, int n,
          StepConst c, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    float4 vv = v[i];
    const float4 p = x[i];
    vv.x = ffma(c.gravx, c.dt, vv.x);
    vv.y = ffma(c.gravy, c.dt, vv.y);
    vv.z = ffma(c.gravz, c.dt, vv.z);
    float4 q;
    q.x = ffma(vv.x, c.dt, p.x);
    q.y = ffma(vv.y, c.dt, p.y);
    q.z = ffma(vv.z, c.dt, p.z);
    q.w = p.w;
    xs[i] = q;
    vin[i] = vv;
    GridConst g;
    uint32_t base;
    grid_of<B>(c, i, g, base);
    put_key(keys, bins, i, base + key_of(g, q));
}

__global__ void __launch_bounds__(kBlock)
k_cell_ranges(const uint32_t* __restrict__ skeys, int* __restrict__ cs, int* __restrict__ ce,
              int n, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    const uint32_t key = skeys[i];
    if (i == 0 || skeys[i - 1] != key) cs[key] = i;
    if (i == n - 1 || skeys[i + 1] != key) ce[key] = i + 1;
}

// first[k] = lower_bound(sorted keys, k) for k in [0, cells]: the particles of
// cells [a, b] are exactly [first[a], first[b + 1]).  Equivalent to the
// reference's cellStart/cellEnd pair (spatial_grid.cu:123-137) with empty
// cells resolved to the next occupied one, so a run of cells along x is one
// contiguous index range.
__global__ void __launch_bounds__(kBlock)
k_gather_xs(const uint32_t* __restrict__ perm, const float4* __restrict__ xs_in,
            float4* __restrict__ xs_out, const uint32_t* __restrict__ org_in,
            uint32_t* __restrict__ org_out, float* __restrict__ sx, float* __restrict__ sy,
            float* __restrict__ sz, int n, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    const uint32_t p = perm[i];
    const float4 q = xs_in[p];
    xs_out[i] = q;
    sx[i] = q.x;
    sy[i] = q.y;
    sz[i] = q.z;
    if (org_out) org_out[i] = org_in ? org_in[p] : p;
}

// Lower bound of key k in skeys[0, n), searched outward from a guess: the
// table of the previous rebuild, whose entries move little between
// iterations.  Any guess gives the same answer; a good one needs one or two
// loads instead of log2(n).
__device__ __forceinline__ int lower_bound_from(const uint32_t* __restrict__ skeys, int n,
                                                uint32_t k, int guess) {
    int g = min(max(guess, 0), n);
    int lo, hi;  // answer in [lo, hi]
    if (g > 0 && __ldg(&skeys[g - 1]) >= k) {
        // Answer < g: gallop down until skeys[lo - 1] < k (or lo == 0).
        hi = g - 1;
        int step = 1;
        lo = g - 1;
        while (lo > 0 && __ldg(&skeys[lo - 1]) >= k) {
            hi = lo - 1;
            lo = lo > step ? lo - step : 0;
            step = step < (1 << 29) ? step << 1 : step;
        }
    } else if (g < n && __ldg(&skeys[g]) < k) {
        // Answer > g: gallop up until skeys[hi] >= k (or hi == n).
        lo = g + 1;
        int step = 1;
        hi = min(n, g + 1);
        while (hi < n && __ldg(&skeys[hi]) < k) {
            lo = hi + 1;
            hi = n - hi > step ? hi + step : n;
            step = step < (1 << 29) ? step << 1 : step;
        }
    } else {
        return g;
    }
    // Invariant: skeys[lo - 1] < k (or lo == 0) and skeys[hi] >= k (or hi == n).
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&skeys[mid]) < k) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// One launch after each sort: thread i reorders particle i (as k_gather_xs)
// and refreshes first[i] for i <= cells, in place.
__global__ void __launch_bounds__(kBlock)
k_gather_first(const uint32_t* __restrict__ perm, const float4* __restrict__ xs_in,
               float4* __restrict__ xs_out, const uint32_t* __restrict__ org_in,
               uint32_t* __restrict__ org_out, float* __restrict__ sx, float* __restrict__ sy,
               float* __restrict__ sz, int n, const uint32_t* __restrict__ skeys, uint32_t cells,
               int* __restrict__ first, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (fatal(status)) return;
    if (i < n) {
        const uint32_t p = perm[i];
        const float4 q = xs_in[p];
        xs_out[i] = q;
        sx[i] = q.x;
        sy[i] = q.y;
        sz[i] = q.z;
        org_out[i] = org_in ? org_in[p] : p;
    }
    if (static_cast<uint32_t>(i) <= cells) {
        const uint32_t k = static_cast<uint32_t>(i);
        first[k] = lower_bound_from(skeys, n, k, first[k]);
    }
}

// ---------------------------------------------------------------------------
// Neighbour walk.  Order of the list = z -> y -> x over the clamped cells,
// ascending sorted index inside a cell, self skipped, accept d2 <= h2
// (src/pbf/neighbors.cu:52-86).  With LAMBDA the constraint terms of
// computeLambda are accumulated in that same list order.
// ---------------------------------------------------------------------------
// Two neighbours' terms, lane 0 first: the same sums as two lambda_add calls.
__device__ __forceinline__ void lambda_add2(const KernelConst& k, LambdaAcc& a, f32x2 dx, f32x2 dy,
                                            f32x2 dz, f32x2 d2) {
    const f32x2 s = spiky_scale2(k, d2);
    float w0, w1, x0, x1, y0, y1, z0, z1;
    unpack2(poly6_2(k, d2), w0, w1);
    unpack2(mul2(dx, s), x0, x1);
    unpack2(mul2(dy, s), y0, y1);
    unpack2(mul2(dz, s), z0, z1);
    a.wsum = fadd(fadd(a.wsum, w0), w1);
    a.s2 = ffma(z0, z0, ffma(y0, y0, ffma(x0, x0, a.s2)));
    a.s2 = ffma(z1, z1, ffma(y1, y1, ffma(x1, x1, a.s2)));
    a.gx = fadd(fadd(a.gx, x0), x1);
    a.gy = fadd(fadd(a.gy, y0), y1);
    a.gz = fadd(fadd(a.gz, z0), z1);
}

// Bits of a 32-candidate chunk from j0 (the highest: candidate j0) that belong
// to the row range [s, e), less the particle i itself.
__device__ __forceinline__ uint32_t chunk_valid(int j0, int s, int e, int i) {
    // Shifts clamp at 32: all or nothing past the chunk's ends.
    const uint32_t past = __funnelshift_rc(0xffffffffu, 0u, e - j0);
    const uint32_t self = __funnelshift_rc(0x80000000u, 0u, static_cast<uint32_t>(i - j0));
    const uint32_t valid = (0xffffffffu >> max(s - j0, 0)) & ~(past | self);
    return valid;
}

// Tests the chunk from j0 four candidates at a time, as far as the range reaches
// (left candidates): a row of some 20 candidates seldom fills 32.  Tested 16 / 8
// / 4 at a time walk and lambda take 231 / 212 / 206 us at 1,048,576 particles, 65
// / 61 / 58 at 262,144 and 695 / 682 / 688 for 256 batched scenes.
template <int K, class Test>
__device__ __forceinline__ void test_groups(Test test4, int j0, int left, uint32_t& acc) {
    test4(j0 + K, acc);
    if constexpr (K < 28) {
        if (left <= K + 4) acc <<= 28 - K;
        else test_groups<K + 4>(test4, j0, left, acc);
    }
}

// The hits of particle i (position pi) chunk by chunk, in list order:
// hits(j0, bits) for each 32-candidate chunk from j0 (the highest bit is
// candidate j0).
//
// Rows z -> y, each one index range walked in ascending order -- exactly the
// reference's z -> y -> x cell walk (neighbors.cu:52-86).  Each range is
// tested in 32-candidate chunks from a multiple of 4; candidates outside [s, e)
// and the particle itself are masked off.  The component arrays are padded
// (soa_stride_for), so a chunk may read past the last particle.  All lanes of
// the warp take every row and chunk step together (active: the lane has a
// particle), and hits is called by all of them.
template <bool B, bool WIDE, class Hits>
__device__ __forceinline__ void for_each_chunk(const StepConst& c, int i, bool active, float4 pi,
                                               const float* __restrict__ sx,
                                               const float* __restrict__ sy,
                                               const float* __restrict__ sz,
                                               const int* __restrict__ first, Hits hits) {
    const StencilRows<B> rows(c, i, pi);
    // The hit test d2 <= h2 as a sign bit: for finite d2 it holds exactly
    // when d2 - h2u < 0, h2u being the float just above h2 (the difference
    // of two distinct floats is never zero, and +inf or NaN, the canonical
    // NaN of the FP32 units, give a clear sign bit: no hit, as d2 <= h2).
    const f32x2 h2u = splat2(__uint_as_float(__float_as_uint(c.k.h2) + 1u));
    const f32x2 px = splat2(pi.x), py = splat2(pi.y), pz = splat2(pi.z);
    // 4 candidates from j (a multiple of 4): the x, y, z arrays are read
    // four floats at a time and tested two at a time with FP32x2
    // arithmetic; each test's sign bit is shifted into acc (the first
    // candidate ends up highest).
    auto test4 = [&](int j, uint32_t& acc) {
        const float4 X = __ldg(reinterpret_cast<const float4*>(sx + j));
        const float4 Y = __ldg(reinterpret_cast<const float4*>(sy + j));
        const float4 Z = __ldg(reinterpret_cast<const float4*>(sz + j));
        const f32x2 da = dist2x2(sub2(px, pack2(X.x, X.y)), sub2(py, pack2(Y.x, Y.y)),
                                 sub2(pz, pack2(Z.x, Z.y)));
        const f32x2 db = dist2x2(sub2(px, pack2(X.z, X.w)), sub2(py, pack2(Y.z, Y.w)),
                                 sub2(pz, pack2(Z.z, Z.w)));
        float a0, a1, b0, b1;
        unpack2(sub2(da, h2u), a0, a1);
        unpack2(sub2(db, h2u), b0, b1);
        acc = __funnelshift_l(__float_as_uint(a0), acc, 1);
        acc = __funnelshift_l(__float_as_uint(a1), acc, 1);
        acc = __funnelshift_l(__float_as_uint(b0), acc, 1);
        acc = __funnelshift_l(__float_as_uint(b1), acc, 1);
    };
    // Steps of the warp: the largest radius of its scenes.  WIDE (a stage call's
    // radius of several cells, one grid): as far as the grid has rows, or a radius
    // that reaches far past a thin grid would never end.  With the step's radius of
    // one cell two bounds cost 0.2 to 0.4 % of a frame and save 1 % where the grid
    // is one cell thick.
    int Rz, Ry;
    if constexpr (WIDE) {
        Rz = min(rows.g.radius, rows.g.gz - 1);
        Ry = min(rows.g.radius, rows.g.gy - 1);
    } else {
        Rz = Ry = __reduce_max_sync(0xffffffffu, rows.g.radius);
    }
    for (int dz = -Rz; dz <= Rz; ++dz)
        for (int dy = -Ry; dy <= Ry; ++dy) {
            const int z = rows.cz + dz, y = rows.cy + dy;
            int s = 0, e = 0;
            if (!active || z < rows.z0 || z > rows.z1 || y < rows.y0 || y > rows.y1 ||
                !rows.range(first, z, y, s, e))
                s = e = 0;
            for (int j0 = s & ~3; __any_sync(0xffffffffu, j0 < e); j0 += 32) {
                const int left = e - j0;
                uint32_t acc = 0u;
                if (left > 0) {
                    test_groups<0>(test4, j0, left, acc);
                    acc &= chunk_valid(j0, s, e, i);
                }
                hits(j0, acc);
            }
        }
}

// Compact lists.  The lists of a warp's 32 particles share a slice as wide as
// the longest of them, entry after entry (offset 32 w + lane, step 32): the 32
// threads that read entry k of their lists read 128 bytes in a row, as with
// slot-major lists.  Back to back (step 1) they read 32 sectors: delta p 148
// against 98 us, vorticity 188 against 137, confinement 170 against 123 at
// 1,048,576 particles.  The walks take the slices one after another as they go
// (c.nb_ctl counts the entries), so that no pass has to count the neighbours
// first: frame 17.96 ms with a walk that counts and a scan before each walk,
// 13.84 without, at 8,388,608 particles; 2.37 and 1.78 at 1,048,576.  The slices
// of the scenes here take a tenth to a third more entries than the lists.  When
// they do not fit, the rebuild starts over: counts, a scan of them, and the walk
// into lists back to back (or in slices where those fit after all); the frame's
// later rebuilds then go that way at once (1,048,576 particles 3.00 ms with 4 %
// more capacity than the lists take).
constexpr size_t kNoPlace = ~size_t(0);
constexpr int kCtlUsed = 0, kCtlFailed = 2, kCtlScanned = 3;  // words of c.nb_ctl

// The first entry of the lane's list, in a slice for the longest of the warp's.
__device__ __forceinline__ size_t alloc_lists(const StepConst& c, int count) {
    const int lane = threadIdx.x & 31;
    const unsigned need = 32u * __reduce_max_sync(0xffffffffu, static_cast<unsigned>(count));
    unsigned long long at = 0ull;
    if (lane == 0)
        at = atomicAdd(reinterpret_cast<unsigned long long*>(c.nb_ctl + kCtlUsed),
                       static_cast<unsigned long long>(need));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (at + need > c.nb_cap) {
        if (lane == 0) c.nb_ctl[kCtlFailed] = 1u;
        return kNoPlace;
    }
    return static_cast<size_t>(at) + lane;
}

// Whether the walk that allocates does nothing; thread 0 of the grid sets the
// slices' step.
__device__ __forceinline__ bool skip_alloc(const StepConst& c) {
    const bool skip = !c.nb_retry && __ldcg(&c.nb_ctl[kCtlScanned]) != 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (skip) c.nb_ctl[kCtlFailed] = 1u;
        else *c.nb_step = 32u;
    }
    return skip;
}

// Whether the walk into scanned offsets does nothing.
__device__ __forceinline__ bool skip_scanned(const StepConst& c) {
    if (c.nb_off == nullptr) return false;  // slot-major lists
    if (blockIdx.x == 0 && threadIdx.x == 0) c.nb_ctl[kCtlFailed] = 0u;
    return __ldcg(&c.nb_ctl[kCtlScanned]) == 0u;
}

// Entries of a lane's queue of chunks with hits (8 bytes each, in shared
// memory).  A stencil of nine rows with some 20 candidates each has 9 to 11 such
// chunks; search time at 10 / 12 / 16 entries: 0.930 / 0.923 / 0.928 ms at
// 1,048,576 particles, 10.56 / 10.41 / 10.42 for 8,388,608 in dense blobs.
constexpr int kQueue = 12;
inline size_t queue_bytes(int threads) { return sizeof(uint2) * kQueue * threads; }

// The neighbour walk of particle i with the terms of its neighbours: writes the
// list into nbr (at most cap entries), hands the neighbours over in list order
// (load, use2, use1 as for for_each_neighbor_pair) and returns the full count.
// ALLOC: the warp takes the place of its lists (see alloc_lists) once it knows
// their lengths, in the first walk when the queues held all hits, else before a
// second; -1 if there is no place left.
//
// Bound by issue (67 % active, FP32x2 operations taking two slots) and the L1's
// data pipe (77 %: 12 bytes a lane for each candidate).  Appending the hits of
// each chunk at once costs a warp the largest number of hits of any lane, chunk
// by chunk (2 to 3 times the average), and the terms need a second pass over the
// list.  So the chunks with hits are queued, and the lanes take their neighbours
// from their queues one by one, in step: list entry and terms in one loop whose
// length is the largest neighbour count.  The queues are emptied together when
// any is full (lanes that empty theirs by themselves: walk 30 to 80 % longer in
// dense scenes).  Walk and lambda, before and with all of this: 38 -> 28 us at
// 65,536 particles, 76 -> 58 at 262,144, 280 -> 206 at 1,048,576 and 875 -> 688
// for 256 batched scenes; the final walk with XSPH at 1,048,576 310 -> 248 (at 72
// registers, with 4 to 12 bytes of spills; at 64 with more of them: +3 %).
template <bool B, bool ALLOC, bool WIDE, class T, class Load, class Use2, class Use1>
__device__ __forceinline__ int walk_terms(const StepConst& c, int i, bool active, float4 pi,
                                          const float* __restrict__ sx,
                                          const float* __restrict__ sy,
                                          const float* __restrict__ sz,
                                          const int* __restrict__ first,
                                          uint32_t* __restrict__ nbr, int cap, Load load,
                                          Use2 use2, Use1 use1) {
    extern __shared__ uint2 queues[];
    uint2* const queue = queues + threadIdx.x;
    const int step = blockDim.x;
    uint32_t* __restrict__ out = ALLOC ? nbr : nbr + nb_first(c, i);
    const size_t stride = ALLOC ? 32 : nb_step(c);
    bool placed = !ALLOC;  // out is known
    bool over = false;     // hits left out of the queue
    int steps = 0;         // chunks since the queue was empty
    int count = 0;         // neighbours handed over
    int found = 0;         // neighbours in the queue
    uint2* tail = queue;
    const uint2* const end_of_queue = queue + kQueue * step;
    auto drain = [&]() {
        const uint2* head = queue;
        uint32_t bits = 0u, j0 = 0u;
        uint32_t* at = out + static_cast<size_t>(count) * stride;
        auto pop = [&]() {
            if (!bits) {
                const uint2 q = *head;
                head += step;
                j0 = q.x;
                bits = q.y;
            }
            const int b = 31 - __clz(bits);
            bits ^= 1u << b;
            const uint32_t j = j0 - b;
            *at = j;
            at += stride;
            return j;
        };
        int left = min(found, cap - count);
        for (; left >= 2; left -= 2) {
            const T a = load(pop()), b = load(pop());
            use2(a, b);
        }
        if (left > 0) use1(load(pop()));
        count += found;
        tail = queue;
        found = 0;
        steps = 0;
    };
#pragma unroll 1
    for (;;) {
        for_each_chunk<B, WIDE>(c, i, active, pi, sx, sy, sz, first, [&](int j0, uint32_t bits) {
            if (bits) {
                if (!ALLOC || tail != end_of_queue) {
                    *tail = make_uint2(static_cast<uint32_t>(j0) + 31u, bits);
                    tail += step;
                } else {
                    over = true;
                }
                found += __popc(bits);
            }
            if (placed && (ALLOC || ++steps >= kQueue) && __any_sync(0xffffffffu, tail == end_of_queue)) drain();
        });
        if (placed) break;
        const size_t at = alloc_lists(c, min(found, cap));
        if (at == kNoPlace) return -1;
        out = nbr + at;
        if (active) c.nb_off[i] = static_cast<uint32_t>(at);
        placed = true;
        if (!__any_sync(0xffffffffu, over)) break;
        tail = queue;
        found = 0;
    }
    drain();
    return count;
}

template <bool LAMBDA, bool B, bool ALLOC, bool WIDE = false>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_search(const float4* __restrict__ xs, const float* __restrict__ sx,
         const float* __restrict__ sy, const float* __restrict__ sz, const int* __restrict__ first,
         StepConst c, int n, uint32_t* __restrict__ nbr, int* __restrict__ cnt,
         float* __restrict__ lam, unsigned* __restrict__ status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (__any_sync(0xffffffffu, fatal(status))) return;
    if (ALLOC ? skip_alloc(c) : skip_scanned(c)) return;
    const bool active = i < n;
    i = min(i, n - 1);
    const float4 pi = xs[i];
    const f32x2 px = splat2(pi.x), py = splat2(pi.y), pz = splat2(pi.z);
    LambdaAcc acc{c.k.c_poly6, 0.0f, 0.0f, 0.0f, 0.0f};
    const int count = walk_terms<B, ALLOC, WIDE, float4>(
        c, i, active, pi, sx, sy, sz, first, nbr, c.max_nb,
        [&](uint32_t j) { return LAMBDA ? __ldg(&xs[j]) : float4{}; },
        [&](const float4& a, const float4& b) {
            if (!LAMBDA) return;
            const f32x2 dx = sub2(px, pack2(a.x, b.x));
            const f32x2 dy = sub2(py, pack2(a.y, b.y));
            const f32x2 dz = sub2(pz, pack2(a.z, b.z));
            lambda_add2(c.k, acc, dx, dy, dz, dist2x2(dx, dy, dz));
        },
        [&](const float4& a) {
            if (!LAMBDA) return;
            const float dx = fsub(pi.x, a.x), dy = fsub(pi.y, a.y), dz = fsub(pi.z, a.z);
            lambda_add(c.k, acc, dx, dy, dz, dist2(dx, dy, dz));
        });
    if (!active || count < 0) return;
    cnt[i] = count;
    if (count > c.max_nb) atomicOr(status, kStatusNeighborOverflow);
    if (LAMBDA) lam[i] = count > c.max_nb ? CUDART_NAN_F : lambda_of_acc<B>(c, i, acc);
}

// Compact lists that start over: the walk's neighbour count only.
template <bool B>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_count(const float4* __restrict__ xs, const float* __restrict__ sx,
        const float* __restrict__ sy, const float* __restrict__ sz,
        const int* __restrict__ first, StepConst c, int n, int* __restrict__ cnt,
        unsigned* __restrict__ status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (__any_sync(0xffffffffu, fatal(status))) return;
    if (i < 2) c.nb_ctl[kCtlUsed + i] = 0u;  // for the next rebuild
    if (__ldcg(&c.nb_ctl[kCtlFailed]) == 0u) return;
    const bool active = i < n;
    i = min(i, n - 1);
    int count = 0;
    for_each_chunk<B, false>(c, i, active, xs[i], sx, sy, sz, first,
                      [&](int, uint32_t bits) { count += __popc(bits); });
    if (!active) return;
    cnt[i] = count;
    if (count > c.max_nb) atomicOr(status, kStatusNeighborOverflow);
}

// Exclusive scan of the counts into list offsets, in two launches: tile totals,
// and the offsets.  64-bit sums; offsets are 32-bit because the list capacity is
// below 2^32.
constexpr int kScanThreads = 256, kScanItems = 8, kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ unsigned long long block_scan_u64(unsigned long long v,
                                                             unsigned long long* warp_tot,
                                                             unsigned long long& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x / 32;
        unsigned long long w = lane < nw ? warp_tot[lane] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) warp_tot[lane] = w;
    }
    __syncthreads();
    total = warp_tot[blockDim.x / 32 - 1];
    const unsigned long long before = warp ? warp_tot[warp - 1] : 0ull;
    __syncthreads();
    return before + incl - v;
}

// The thread's kScanItems consecutive counts, and the entries of its slice
// (on the slice's first thread, 0 on the others).
__device__ __forceinline__ void load_list_counts(const int* __restrict__ cnt, int n, int base,
                                                 unsigned (&v)[kScanItems],
                                                 unsigned long long& sum,
                                                 unsigned long long& slice) {
    unsigned widest = 0u;
    sum = 0ull;
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        v[r] = base + r < n ? static_cast<unsigned>(max(0, cnt[base + r])) : 0u;
        sum += v[r];
        widest = max(widest, v[r]);
    }
#pragma unroll
    for (int o = 1; o < 32 / kScanItems; o <<= 1)
        widest = max(widest, __shfl_xor_sync(0xffffffffu, widest, o));
    slice = threadIdx.x % (32 / kScanItems) == 0 ? 32ull * widest : 0ull;
}

// sums: the tiles' entries back to back, their total, then the same in slices.
__global__ void __launch_bounds__(kScanThreads)
k_nb_scan_tiles(const int* __restrict__ cnt, int n, unsigned long long* __restrict__ sums,
                int tiles, const unsigned* __restrict__ ctl,
                const unsigned* __restrict__ status) {
    __shared__ unsigned long long warp_tot[kScanThreads / 32];
    if (__syncthreads_or(fatal(status) || __ldcg(&ctl[kCtlFailed]) == 0u)) return;
    unsigned v[kScanItems];
    unsigned long long sum, slice, total, total_sliced;
    load_list_counts(cnt, n, blockIdx.x * kScanTile + threadIdx.x * kScanItems, v, sum, slice);
    block_scan_u64(sum, warp_tot, total);
    block_scan_u64(slice, warp_tot, total_sliced);
    if (threadIdx.x == 0) {
        sums[blockIdx.x] = total;
        sums[tiles + 1 + blockIdx.x] = total_sliced;
    }
}

// The offsets and the step between entries, and the capacity check.
__global__ void __launch_bounds__(kScanThreads)
k_nb_scan_add(const int* __restrict__ cnt, int n, size_t cap,
              const unsigned long long* __restrict__ sums, int tiles, uint32_t* __restrict__ off,
              uint32_t* __restrict__ step, unsigned* __restrict__ ctl,
              unsigned* __restrict__ status) {
    __shared__ unsigned long long warp_tot[kScanThreads / 32];
    const bool skip = __ldcg(&ctl[kCtlFailed]) == 0u;
    if (__syncthreads_or(fatal(status))) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) ctl[kCtlScanned] = skip ? 0u : 1u;
    if (__syncthreads_or(skip)) return;
    // Every block sums the tiles: before its own and in all, each way.
    unsigned long long before[2] = {0ull, 0ull}, all[2] = {0ull, 0ull}, start[2], total[2];
    for (int t = threadIdx.x; t < tiles; t += kScanThreads)
#pragma unroll
        for (int way = 0; way < 2; ++way) {
            const unsigned long long s = sums[way * (tiles + 1) + t];
            all[way] += s;
            if (t < static_cast<int>(blockIdx.x)) before[way] += s;
        }
#pragma unroll
    for (int way = 0; way < 2; ++way) {
        block_scan_u64(before[way], warp_tot, start[way]);
        block_scan_u64(all[way], warp_tot, total[way]);
    }
    const bool sliced = total[1] <= cap;
    const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
    unsigned v[kScanItems];
    unsigned long long sum, slice, tile;
    load_list_counts(cnt, n, base, v, sum, slice);
    unsigned long long run =
        block_scan_u64(sliced ? slice : sum, warp_tot, tile) + start[sliced ? 1 : 0];
    // A slice's first thread holds its start; the others' exclusive sums are
    // past it.
    if (sliced) run = __shfl_sync(0xffffffffu, run, threadIdx.x & 31 & ~(32 / kScanItems - 1));
#pragma unroll
    for (int r = 0; r < kScanItems; ++r) {
        const unsigned long long o = sliced ? run + ((base + r) & 31) : run;
        // A clamped offset means a total above any capacity, flagged below.
        if (base + r < n) off[base + r] = static_cast<uint32_t>(min(o, 0xffffffffull));
        if (!sliced) run += v[r];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *step = sliced ? 32u : 1u;
        if (total[0] > cap) atomicOr(status, kStatusListOverflow);
    }
}

// Walks a slot-major list in order, four neighbours at a time: their four
// gathers (load(j)) are issued before any term is used.  Terms are handed
// over two at a time (use2(first, second)) for FP32x2 evaluation; a last odd
// neighbour goes to use1.  List order is kept.
template <class T, class Load, class Use2, class Use1>
__device__ __forceinline__ void for_each_neighbor_pair(const uint32_t* __restrict__ row,
                                                       size_t stride, int count, Load load,
                                                       Use2 use2, Use1 use1) {
    // The indices of the next four neighbours are loaded while the current
    // four are gathered and used, so the list read (from DRAM) overlaps the
    // dependent gathers instead of preceding them.
    int k = 0;
    uint32_t jn[4];
    if (count >= 4) {
#pragma unroll
        for (int b = 0; b < 4; ++b) jn[b] = __ldg(&row[static_cast<size_t>(b) * stride]);
    }
    for (; k + 4 <= count; k += 4) {
        uint32_t j[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) j[b] = jn[b];
        if (k + 8 <= count) {
#pragma unroll
            for (int b = 0; b < 4; ++b)
                jn[b] = __ldg(&row[static_cast<size_t>(k + 4 + b) * stride]);
        }
        T v[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) v[b] = load(j[b]);
        use2(v[0], v[1]);
        use2(v[2], v[3]);
    }
    if (k + 2 <= count) {
        const uint32_t j0 = __ldg(&row[static_cast<size_t>(k) * stride]);
        const uint32_t j1 = __ldg(&row[static_cast<size_t>(k + 1) * stride]);
        const T a = load(j0), b = load(j1);
        use2(a, b);
        k += 2;
    }
    if (k < count) use1(load(__ldg(&row[static_cast<size_t>(k) * stride])));
}

struct PosVel {
    float4 p, v;
};
struct PosLam {
    float4 p;
    float l;
};

// Differences a - (b0, b1) of one float against a pair.
__device__ __forceinline__ f32x2 diff2(float a, float b0, float b1) {
    return sub2(splat2(a), pack2(b0, b1));
}
__device__ __forceinline__ f32x2 rdiff2(float b0, float b1, float a) {
    return sub2(pack2(b0, b1), splat2(a));
}
// crossc on pairs: a.y*b.z - a.z*b.y with one rounding of a.y*b.z.
__device__ __forceinline__ f32x2 crossc2(f32x2 ay, f32x2 az, f32x2 by, f32x2 bz) {
    return fma2(ay, bz, mul2(mul2(az, splat2(-1.0f)), by));
}

// computeDeltaPosition summed in list order (pbf_solver_kernels.cu:134-171).
// Indices, positions and lambdas of four neighbours are loaded before any of
// them is used, so the dependent gathers overlap; the sum stays in list order.
template <int N>
__device__ __forceinline__ void delta_term(const StepConst& c, float4 pi, float li, float4 pj,
                                           float lj, float& ax, float& ay, float& az) {
    const float dx = fsub(pi.x, pj.x), dy = fsub(pi.y, pj.y), dz = fsub(pi.z, pj.z);
    const float d2 = dist2(dx, dy, dz);
    float gx, gy, gz;
    spiky(c.k, dx, dy, dz, d2, gx, gy, gz);
    const float ls = fadd(fadd(li, lj), scorr<N>(c.sc, d2));
    ax = ffma(ls, gx, ax);
    ay = ffma(ls, gy, ay);
    az = ffma(ls, gz, az);
}

// Two neighbours' terms, lane 0 first: the same sums as two delta_term calls.
template <int N>
__device__ __forceinline__ void delta_term2(const StepConst& c, float4 pi, float li, float4 pa,
                                            float la, float4 pb, float lb, float& ax, float& ay,
                                            float& az) {
    const f32x2 dx = sub2(splat2(pi.x), pack2(pa.x, pb.x));
    const f32x2 dy = sub2(splat2(pi.y), pack2(pa.y, pb.y));
    const f32x2 dz = sub2(splat2(pi.z), pack2(pa.z, pb.z));
    const f32x2 d2 = dist2x2(dx, dy, dz);
    const f32x2 s = spiky_scale2(c.k, d2);
    const f32x2 ls = add2(add2(splat2(li), pack2(la, lb)), scorr2<N>(c.sc, d2));
    float l0, l1, x0, x1, y0, y1, z0, z1;
    unpack2(ls, l0, l1);
    unpack2(mul2(dx, s), x0, x1);
    unpack2(mul2(dy, s), y0, y1);
    unpack2(mul2(dz, s), z0, z1);
    ax = ffma(l1, x1, ffma(l0, x0, ax));
    ay = ffma(l1, y1, ffma(l0, y0, ay));
    az = ffma(l1, z1, ffma(l0, z0, az));
}

template <int N>
__device__ __forceinline__ void delta_sum(const StepConst& c, const float4* __restrict__ xs,
                                          const uint32_t* __restrict__ nbr,
                                          const float* __restrict__ lam, int i, int count,
                                          float4 pi, float gs, float& dpx, float& dpy,
                                          float& dpz) {
    const float li = lam[i];
    float ax = 0.0f, ay = 0.0f, az = 0.0f;
    for_each_neighbor_pair<PosLam>(
        nbr + nb_first(c, i), nb_step(c), count,
        [&](uint32_t j) { return PosLam{__ldg(&xs[j]), __ldg(&lam[j])}; },
        [&](const PosLam& a, const PosLam& b) {
            delta_term2<N>(c, pi, li, a.p, a.l, b.p, b.l, ax, ay, az);
        },
        [&](const PosLam& q) { delta_term<N>(c, pi, li, q.p, q.l, ax, ay, az); });
    dpx = fmul(gs, ax);
    dpy = fmul(gs, ay);
    dpz = fmul(gs, az);
}

// delta p + applyDeltaPosition + CollisionSystem::solve + next cell keys.
// N: artificial-pressure exponent fixed at compile time (0 = read at run time).
// moved, pre: see apply_delta.
template <int N, bool B>
__global__ void PBF_GATHER_REGS(48)
k_delta_apply(const float4* __restrict__ xs, const uint32_t* __restrict__ nbr,
              const int* __restrict__ cnt, const float* __restrict__ lam, StepConst c, int n,
              float4* __restrict__ xs_out, uint32_t* __restrict__ keys_out, CellBins bins,
              uint8_t* __restrict__ moved, float4* __restrict__ pre,
              unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    const float4 pi = xs[i];
    const int count = cnt[i];
    float dpx, dpy, dpz;
    if (!count_ok(count, c.max_nb)) {
        dpx = dpy = dpz = CUDART_NAN_F;
    } else {
        const float gs = B ? scene_of(c, i).gs : c.gs;
        delta_sum<N>(c, xs, nbr, lam, i, count, pi, gs, dpx, dpy, dpz);
    }
    apply_delta<B>(c, i, pi, dpx, dpy, dpz, xs_out, keys_out, bins, moved, pre, status);
}

// Gather x, v_in, v.w and ids through the composite permutation of the
// substep, then updateVelocityAndPosition (pbf_solver_kernels.cu:195-211).
// The new positions are the predicted ones, so xs becomes x without a copy.
__global__ void __launch_bounds__(kBlock)
k_finalize(const uint32_t* __restrict__ org, const float4* __restrict__ x_old,
           const float4* __restrict__ vin_old, const float4* __restrict__ v_old,
           const uint32_t* __restrict__ id_old, const float4* __restrict__ xs, int n,
           StepConst c, float4* __restrict__ v_new, float4* __restrict__ vin_new,
           uint32_t* __restrict__ id_new, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    const uint32_t o = org[i];
    const float4 xo = x_old[o];
    const float4 q = xs[i];
    v_new[i] = updated_velocity(xo, q, v_old[o].w, c.inv_dt);
    vin_new[i] = vin_old[o];
    if (id_new) id_new[i] = id_old[o];
}

// applyXsphViscosity (pbf_solver_kernels.cu:213-266).
struct XsphAcc {
    float x, y, z;
};
__device__ __forceinline__ void xsph_add2(const KernelConst& k, XsphAcc& s, float4 pi, float4 vi,
                                          const PosVel& a, const PosVel& b) {
    float w0, w1, x0, x1, y0, y1, z0, z1;
    unpack2(poly6_2(k, dist2x2(diff2(pi.x, a.p.x, b.p.x), diff2(pi.y, a.p.y, b.p.y),
                               diff2(pi.z, a.p.z, b.p.z))),
            w0, w1);
    unpack2(rdiff2(a.v.x, b.v.x, vi.x), x0, x1);
    unpack2(rdiff2(a.v.y, b.v.y, vi.y), y0, y1);
    unpack2(rdiff2(a.v.z, b.v.z, vi.z), z0, z1);
    s.x = ffma(x1, w1, ffma(x0, w0, s.x));
    s.y = ffma(y1, w1, ffma(y0, w0, s.y));
    s.z = ffma(z1, w1, ffma(z0, w0, s.z));
}
__device__ __forceinline__ void xsph_add(const KernelConst& k, XsphAcc& s, float4 pi, float4 vi,
                                         const PosVel& q) {
    const float w = poly6(k, dist2(fsub(pi.x, q.p.x), fsub(pi.y, q.p.y), fsub(pi.z, q.p.z)));
    s.x = ffma(fsub(q.v.x, vi.x), w, s.x);
    s.y = ffma(fsub(q.v.y, vi.y), w, s.y);
    s.z = ffma(fsub(q.v.z, vi.z), w, s.z);
}
__device__ __forceinline__ float4 xsph_finish(float xsph_c, const XsphAcc& s, float4 vi) {
    return make_float4(ffma(xsph_c, s.x, vi.x), ffma(xsph_c, s.y, vi.y), ffma(xsph_c, s.z, vi.z),
                       vi.w);
}

__device__ __forceinline__ float4 xsph_one(const StepConst& c, const float4* __restrict__ x,
                                           const float4* __restrict__ v,
                                           const uint32_t* __restrict__ nbr, int count, int i,
                                           float xsph_c) {
    const float4 vi = v[i];
    if (!count_ok(count, c.max_nb))
        return make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, vi.w);
    const float4 pi = x[i];
    XsphAcc s{0.0f, 0.0f, 0.0f};
    for_each_neighbor_pair<PosVel>(
        nbr + nb_first(c, i), nb_step(c), count,
        [&](uint32_t j) { return PosVel{__ldg(&x[j]), __ldg(&v[j])}; },
        [&](const PosVel& a, const PosVel& b) { xsph_add2(c.k, s, pi, vi, a, b); },
        [&](const PosVel& q) { xsph_add(c.k, s, pi, vi, q); });
    return xsph_finish(xsph_c, s, vi);
}

template <bool B>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_xsph(const float4* __restrict__ x, const float4* __restrict__ v,
       const uint32_t* __restrict__ nbr, const int* __restrict__ cnt, StepConst c, int n,
       float4* __restrict__ v_out, const float4* __restrict__ vin, bool resolve,
       const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    float4 out = xsph_one(c, x, v, nbr, cnt[i], i, B ? scene_of(c, i).xsph_c : c.xsph_c);
    if (resolve)
        resolve_velocity(colliders_of<B>(c, i), c.particle_radius, c.restitution, c.friction,
                         x[i], vin[i], out);
    v_out[i] = out;
}

// The final rebuild's walk with applyXsphViscosity fused in (velocities v are
// the updated ones, computed before this walk), and with the velocity response
// when no vorticity pass follows.
template <bool B, bool ALLOC>
__global__ void PBF_GATHER_REGS(72)
k_search_xsph(const float4* __restrict__ xs, const float* __restrict__ sx,
              const float* __restrict__ sy, const float* __restrict__ sz,
              const int* __restrict__ first, StepConst c, int n, uint32_t* __restrict__ nbr,
              int* __restrict__ cnt, const float4* __restrict__ v, float4* __restrict__ v_out,
              const float4* __restrict__ vin, bool resolve, unsigned* __restrict__ status) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (__any_sync(0xffffffffu, fatal(status))) return;
    if (ALLOC ? skip_alloc(c) : skip_scanned(c)) return;
    const bool active = i < n;
    i = min(i, n - 1);
    const float4 pi = xs[i], vi = v[i];
    XsphAcc s{0.0f, 0.0f, 0.0f};
    const int count = walk_terms<B, ALLOC, false, PosVel>(
        c, i, active, pi, sx, sy, sz, first, nbr, c.max_nb,
        [&](uint32_t j) { return PosVel{__ldg(&xs[j]), __ldg(&v[j])}; },
        [&](const PosVel& a, const PosVel& b) { xsph_add2(c.k, s, pi, vi, a, b); },
        [&](const PosVel& q) { xsph_add(c.k, s, pi, vi, q); });
    if (!active || count < 0) return;
    cnt[i] = count;
    if (count > c.max_nb) atomicOr(status, kStatusNeighborOverflow);
    float4 out = count > c.max_nb
                     ? make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, vi.w)
                     : xsph_finish(B ? scene_of(c, i).xsph_c : c.xsph_c, s, vi);
    if (resolve)
        resolve_velocity(colliders_of<B>(c, i), c.particle_radius, c.restitution, c.friction,
                         pi, vin[i], out);
    v_out[i] = out;
}

// computeVorticity (pbf_solver_kernels.cu:268-315).
__global__ void __launch_bounds__(kMaxTunedBlock)
k_vorticity(const float4* __restrict__ x, const float4* __restrict__ v,
            const uint32_t* __restrict__ nbr, const int* __restrict__ cnt, StepConst c, int n,
            float4* __restrict__ omega, bool store_norm, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    const int count = cnt[i];
    if (!count_ok(count, c.max_nb)) {
        omega[i] = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F,
                               store_norm ? CUDART_NAN_F : 0.0f);
        return;
    }
    const float4 pi = x[i], vi = v[i];
    float ox = 0.0f, oy = 0.0f, oz = 0.0f;
    for_each_neighbor_pair<PosVel>(
        nbr + nb_first(c, i), nb_step(c), count,
        [&](uint32_t j) { return PosVel{__ldg(&x[j]), __ldg(&v[j])}; },
        [&](const PosVel& a, const PosVel& b) {
            const f32x2 dx = diff2(pi.x, a.p.x, b.p.x), dy = diff2(pi.y, a.p.y, b.p.y),
                        dz = diff2(pi.z, a.p.z, b.p.z);
            const f32x2 sc = spiky_scale2(c.k, dist2x2(dx, dy, dz));
            const f32x2 gx = mul2(dx, sc), gy = mul2(dy, sc), gz = mul2(dz, sc);
            const f32x2 vx = rdiff2(a.v.x, b.v.x, vi.x), vy = rdiff2(a.v.y, b.v.y, vi.y),
                        vz = rdiff2(a.v.z, b.v.z, vi.z);
            float x0, x1, y0, y1, z0, z1;
            unpack2(crossc2(gy, gz, vy, vz), x0, x1);
            unpack2(crossc2(gz, gx, vz, vx), y0, y1);
            unpack2(crossc2(gx, gy, vx, vy), z0, z1);
            ox = fadd(fadd(ox, x0), x1);
            oy = fadd(fadd(oy, y0), y1);
            oz = fadd(fadd(oz, z0), z1);
        },
        [&](const PosVel& q) {
            const float dx = fsub(pi.x, q.p.x), dy = fsub(pi.y, q.p.y), dz = fsub(pi.z, q.p.z);
            float gx, gy, gz;
            spiky(c.k, dx, dy, dz, dist2(dx, dy, dz), gx, gy, gz);
            const float vx = fsub(q.v.x, vi.x), vy = fsub(q.v.y, vi.y), vz = fsub(q.v.z, vi.z);
            ox = fadd(ox, crossc(gy, gz, vy, vz));
            oy = fadd(oy, crossc(gz, gx, vz, vx));
            oz = fadd(oz, crossc(gx, gy, vx, vy));
        });
    // With store_norm, w carries |omega| (read by the confinement for every
    // neighbour); otherwise w = 0 as computeVorticity writes it.
    omega[i] = make_float4(ox, oy, oz, store_norm ? len3(ox, oy, oz) : 0.0f);
}

// w <- |omega| for a vorticity array written with w = 0.
__global__ void __launch_bounds__(kBlock) k_omega_norm(float4* __restrict__ om, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 w = om[i];
    w.w = len3(w.x, w.y, w.z);
    om[i] = w;
}

// applyVorticityConfinement (pbf_solver_kernels.cu:317-385).
__device__ __forceinline__ float4 confine_one(const StepConst& c, const float4* __restrict__ x,
                                              const uint32_t* __restrict__ nbr, int count,
                                              const float4* __restrict__ om,
                                              const float4* __restrict__ v, int i) {
    const float4 vi = v[i];
    if (!count_ok(count, c.max_nb))
        return make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, vi.w);
    const float4 pi = x[i], wi = om[i];
    const float wil = wi.w;  // |omega_i|, stored by k_vorticity
    float ex = 0.0f, ey = 0.0f, ez = 0.0f;
    for_each_neighbor_pair<PosVel>(
        nbr + nb_first(c, i), nb_step(c), count,
        [&](uint32_t j) { return PosVel{__ldg(&x[j]), __ldg(&om[j])}; },
        [&](const PosVel& a, const PosVel& b) {
            const f32x2 dx = diff2(pi.x, a.p.x, b.p.x), dy = diff2(pi.y, a.p.y, b.p.y),
                        dz = diff2(pi.z, a.p.z, b.p.z);
            const f32x2 sc = spiky_scale2(c.k, dist2x2(dx, dy, dz));
            float m0, m1, x0, x1, y0, y1, z0, z1;
            unpack2(rdiff2(a.v.w, b.v.w, wil), m0, m1);
            unpack2(mul2(dx, sc), x0, x1);
            unpack2(mul2(dy, sc), y0, y1);
            unpack2(mul2(dz, sc), z0, z1);
            ex = ffma(m1, x1, ffma(m0, x0, ex));
            ey = ffma(m1, y1, ffma(m0, y0, ey));
            ez = ffma(m1, z1, ffma(m0, z0, ez));
        },
        [&](const PosVel& q) {
            const float wjl = q.v.w;
            const float dx = fsub(pi.x, q.p.x), dy = fsub(pi.y, q.p.y), dz = fsub(pi.z, q.p.z);
            float gx, gy, gz;
            spiky(c.k, dx, dy, dz, dist2(dx, dy, dz), gx, gy, gz);
            const float md = fsub(wjl, wil);
            ex = ffma(md, gx, ex);
            ey = ffma(md, gy, ey);
            ez = ffma(md, gz, ez);
        });
    return confine_finish(c, ex, ey, ez, wi, vi);
}

template <bool B>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_confine(const float4* __restrict__ x, const uint32_t* __restrict__ nbr,
          const int* __restrict__ cnt, const float4* __restrict__ om,
          const float4* __restrict__ v, StepConst c, int n, float4* __restrict__ v_out,
          const float4* __restrict__ vin, bool resolve, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    float4 out = confine_one(c, x, nbr, cnt[i], om, v, i);
    if (resolve)
        resolve_velocity(colliders_of<B>(c, i), c.particle_radius, c.restitution, c.friction,
                         x[i], vin[i], out);
    v_out[i] = out;
}

template <bool B>
__global__ void __launch_bounds__(kBlock)
k_resolve(const float4* __restrict__ x, const float4* __restrict__ vin, float4* __restrict__ v,
          StepConst c, int n, const unsigned* __restrict__ status) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || fatal(status)) return;
    float4 vv = v[i];
    resolve_velocity(colliders_of<B>(c, i), c.particle_radius, c.restitution, c.friction, x[i],
                     vin[i], vv);
    v[i] = vv;
}

// scatterFloat4ByStableId (pbf_solver_kernels.cu:418-427).  After a run that failed
// the ids may be those of an earlier, larger set of particles, or of none: such
// a value is left out, out holds n.
__global__ void __launch_bounds__(kBlock)
k_scatter_by_id(const float4* __restrict__ vals, const uint32_t* __restrict__ id,
                float4* __restrict__ out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t o = id[i];
    if (o < static_cast<uint32_t>(n)) out[o] = vals[i];
}

__global__ void __launch_bounds__(kBlock) k_iota(uint32_t* a, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = static_cast<uint32_t>(i);
}

// |rho/rho0 - 1| per particle over the current lists.  A run that failed may leave
// counts whose compact lists were never placed or written: entries past the lists'
// capacity or naming no particle slot (of slots) are left out.
__global__ void __launch_bounds__(kBlock)
k_density(const float4* __restrict__ x, const uint32_t* __restrict__ nbr,
          const int* __restrict__ cnt, StepConst c, int n, uint32_t slots,
          float* __restrict__ err) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 pi = x[i];
    const int count = min(cnt[i], c.max_nb);
    float wsum = c.k.c_poly6;
    const size_t list = nb_first(c, i), step = nb_step(c);
    for (int k = 0; k < count; ++k) {
        const size_t at = list + static_cast<size_t>(k) * step;
        if (c.nb_off != nullptr && at >= c.nb_cap) break;
        const uint32_t j = __ldg(&nbr[at]);
        if (j >= slots) continue;
        const float4 pj = __ldg(&x[j]);
        wsum = fadd(wsum, poly6(c.k, dist2(fsub(pi.x, pj.x), fsub(pi.y, pj.y), fsub(pi.z, pj.z))));
    }
    const float mass = c.scenes ? scene_of(c, i).mass : c.mass;
    const float rho0 = c.scenes ? scene_of(c, i).rho0 : c.rho0;
    err[i] = fabsf(fsub(fdiv(fmul(mass, wsum), rho0), 1.0f));
}

// --- stage kernels -----------------------------------------------------------
__global__ void __launch_bounds__(kBlock)
k_grid_keys(const float4* __restrict__ pos, uint32_t* __restrict__ keys, int n, GridConst g) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) keys[i] = key_of(g, pos[i]);
}

__global__ void __launch_bounds__(kBlock)
k_lambda_list(const float4* __restrict__ xs, const uint32_t* __restrict__ nbr,
              const int* __restrict__ cnt, StepConst c, int n, float* __restrict__ lam) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int count = cnt[i];
    if (!count_ok(count, c.max_nb)) {
        lam[i] = CUDART_NAN_F;
        return;
    }
    const float4 pi = xs[i];
    LambdaAcc acc{c.k.c_poly6, 0.0f, 0.0f, 0.0f, 0.0f};
    for (int k = 0; k < count; ++k) {
        const float4 pj = xs[nbr[static_cast<size_t>(k) * c.stride + i]];
        const float dx = fsub(pi.x, pj.x), dy = fsub(pi.y, pj.y), dz = fsub(pi.z, pj.z);
        lambda_add(c.k, acc, dx, dy, dz, dist2(dx, dy, dz));
    }
    lam[i] = lambda_finish(c, acc);
}

__global__ void __launch_bounds__(kBlock)
k_delta_list(const float4* __restrict__ xs, const uint32_t* __restrict__ nbr,
             const int* __restrict__ cnt, const float* __restrict__ lam, StepConst c, int n,
             float4* __restrict__ delta) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int count = cnt[i];
    if (!count_ok(count, c.max_nb)) {
        delta[i] = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, 0.0f);
        return;
    }
    float dx, dy, dz;
    delta_sum<0>(c, xs, nbr, lam, i, count, xs[i], c.gs, dx, dy, dz);
    delta[i] = make_float4(dx, dy, dz, 0.0f);
}

// kind: 0 container, 1 spheres, 2 boxes, 3 planes (one pass), 4 converge all.
__global__ void __launch_bounds__(kBlock)
k_collide(float4* __restrict__ pos, int n, StepConst c, int kind, unsigned* __restrict__ flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 p = pos[i];
    bool mark = false;
    switch (kind) {
        case 0: mark = project_container(c.col, c.particle_radius, p.x, p.y, p.z); break;
        case 1: mark = project_spheres(c.col, c.particle_radius, p.x, p.y, p.z); break;
        case 2: mark = project_boxes(c.col, c.particle_radius, p.x, p.y, p.z); break;
        case 3: mark = project_planes(c.col, c.particle_radius, p.x, p.y, p.z); break;
        default: mark = !project_all(c.col, c.particle_radius, p.x, p.y, p.z); break;
    }
    if (mark) atomicOr(flag, 1u);
    pos[i] = p;
}

__global__ void __launch_bounds__(kBlock)
k_integrate(const float4* __restrict__ x, float4* __restrict__ xs, float4* __restrict__ v,
            int n, StepConst c) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 vv = v[i];
    const float4 p = x[i];
    vv.x = ffma(c.gravx, c.dt, vv.x);
    vv.y = ffma(c.gravy, c.dt, vv.y);
    vv.z = ffma(c.gravz, c.dt, vv.z);
    v[i] = vv;
    xs[i] = make_float4(ffma(vv.x, c.dt, p.x), ffma(vv.y, c.dt, p.y), ffma(vv.z, c.dt, p.z), p.w);
}

}  // namespace

// --- launchers ---------------------------------------------------------------
void launch_predict(const float4* x, const float4* v, float4* xs, float4* vin, uint32_t* keys,
                    const CellBins& bins, int n, const StepConst& c, const unsigned* status,
                    cudaStream_t st) {
    launch_k(c.scenes ? k_predict<true> : k_predict<false>, blocks_for(n), kBlock, st, x, v, xs,
             vin, keys, bins.without_sums(), n, c, status);
}
void launch_cell_ranges(const uint32_t* skeys, int* cs, int* ce, int n, const unsigned* status,
                        cudaStream_t st) {
    k_cell_ranges<<<blocks_for(n), kBlock, 0, st>>>(skeys, cs, ce, n, status);
}
void launch_gather_xs(const uint32_t* perm, const float4* xs_in, float4* xs_out,
                      const uint32_t* org_in, uint32_t* org_out, float* sx, float* sy, float* sz,
                      int n, const unsigned* status, cudaStream_t st) {
    k_gather_xs<<<blocks_for(n), kBlock, 0, st>>>(perm, xs_in, xs_out, org_in, org_out, sx, sy, sz,
                                                  n, status);
}
void launch_gather_first(const uint32_t* perm, const float4* xs_in, float4* xs_out,
                         const uint32_t* org_in, uint32_t* org_out, float* sx, float* sy, float* sz,
                         int n, const uint32_t* skeys, uint64_t cells, int* first,
                         const unsigned* status, cudaStream_t st) {
    const uint64_t threads = std::max<uint64_t>(static_cast<uint64_t>(n), cells + 1);
    launch_k(k_gather_first, blocks_for(threads), kBlock, st, perm, xs_in, xs_out, org_in, org_out,
             sx, sy, sz, n, skeys, static_cast<uint32_t>(cells), first, status);
}
// Lanes per particle of a launch: c.walk_lanes where the group kernels apply.
inline int group_lanes(const StepConst& c, int n) {
    const int L = c.walk_lanes;
    // The walks start 32 threads for three particles.
    if (L < 2 || c.nb_off != nullptr || c.max_nb < L ||
        static_cast<long long>(n) * std::max(L, 11) > (1LL << 30))
        return 1;
    return L;
}

// Threads per block of the neighbour kernels by default.  Smaller blocks even
// out the last wave once there are several blocks an SM: frame at 256 / 128 /
// 64 threads 358 / 329 / 331 us at 131,072 particles, 608 / 593 / 598 at
// 262,144, 1,837 / 1,806 / 1,829 at 1,048,576, 6.70 / 6.66 / 6.68 ms for 256
// batched scenes.  Near the line 256 and 128 threads win in turn, as their blocks
// fill whole waves: 187 / 195 at 24,576, 198 / 202 at 32,768, 204 / 207 at 40,960,
// 214 / 212 at 45,056, 223 / 217 at 57,344, 226 / 231 at 65,536, 260 / 246 at 81,920.
constexpr size_t kBlock128From = 57344;
int default_block(size_t n, int lanes) {
    if (lanes > 1) return kGroupBlock;
    return n >= kBlock128From ? 128 : kBlock;
}
inline int tuned_block(const StepConst& c, int n, int k) {
    return c.blk[k] > 0 ? c.blk[k] : default_block(n, group_lanes(c, n));
}

// Lanes per particle of the neighbour kernels by default (the walks take nine,
// a stencil row each, from 2 on).  Fewer lanes do less work in all, more make
// a shorter launch.  Measured steps of dam breaks in motion at 8 / 16 / 32
// lanes: 98 / 92 / 88 us at 1,024 particles, 108 / 103 / 99 at 2,048, 115 / 109
// / 109 at 4,096, 131 / 128 / 144 at 8,192, 165 / 173 / 193 at 13,824; at 1 / 8
// lanes 178 / 119 at 6,144, 202 / 168 at 13,824, 208 / 177 at 16,384, 200 / 207
// at 20,480 and 194 / 228 at 24,576.
constexpr size_t kLanes32Max = 3072, kLanes16Max = 10240, kLanes8Max = 18432;

int default_walk_lanes(size_t n, int max_nb) {
    int L = n <= kLanes32Max ? 32 : (n <= kLanes16Max ? 16 : (n <= kLanes8Max ? 8 : 1));
    while (L > 1 && max_nb < L) L /= 2;  // a group never has more lanes than list slots
    return L;
}

// The counts and offsets of compact lists, where the walk before found no place
// for its slices.
static void launch_count_and_scan(const float4* xs, const float* sx, const float* sy,
                                  const float* sz, const int* first, const StepConst& c, int n,
                                  int* cnt, unsigned* status, cudaStream_t st) {
    const int bs = tuned_block(c, n, kTunedSearch);
    launch_k(c.scenes ? k_count<true> : k_count<false>, blocks_for(n, bs), bs, st, xs, sx, sy, sz,
             first, c, n, cnt, status);
    const int tiles = static_cast<int>(blocks_for(n, kScanTile));
    launch_k(k_nb_scan_tiles, static_cast<unsigned>(tiles), kScanThreads, st, cnt, n, c.nb_sums,
             tiles, c.nb_ctl, status);
    launch_k(k_nb_scan_add, static_cast<unsigned>(tiles), kScanThreads, st, cnt, n, c.nb_cap,
             c.nb_sums, tiles, c.nb_off, c.nb_step, c.nb_ctl, status);
}

void launch_search(const float4* xs, const float* sx, const float* sy, const float* sz,
                   const int* first, const StepConst& c, int n, uint32_t* nbr, int* cnt, float* lam,
                   unsigned* status, bool with_lambda, cudaStream_t st) {
    const int bs = tuned_block(c, n, with_lambda ? kTunedSearchLambda : kTunedSearch);
    if (group_lanes(c, n) > 1) {
        launch_search_rows(bs, xs, sx, sy, sz, first, c, n, nbr, cnt, lam, status, with_lambda, st);
        return;
    }
    auto walk = [&](auto k) {
        launch_k_smem(k, blocks_for(n, bs), bs, queue_bytes(bs), st, xs, sx, sy, sz, first, c, n,
                      nbr, cnt, lam, status);
    };
    const bool b = c.scenes != nullptr;
    if (c.nb_off) {
        if (with_lambda) walk(b ? k_search<true, true, true> : k_search<true, false, true>);
        else walk(b ? k_search<false, true, true> : k_search<false, false, true>);
        launch_count_and_scan(xs, sx, sy, sz, first, c, n, cnt, status, st);
    }
    if (with_lambda) walk(b ? k_search<true, true, false> : k_search<true, false, false>);
    else if (!b && c.g.radius > 1) walk(k_search<false, false, false, true>);
    else walk(b ? k_search<false, true, false> : k_search<false, false, false>);
}

void launch_search_xsph(const float4* xs, const float* sx, const float* sy, const float* sz,
                        const int* first, const StepConst& c, int n, uint32_t* nbr, int* cnt,
                        const float4* v, float4* v_out, const float4* vin, bool resolve,
                        unsigned* status, cudaStream_t st) {
    const int bs = tuned_block(c, n, kTunedSearch);
    if (group_lanes(c, n) > 1) {
        launch_search_xsph_rows(bs, xs, sx, sy, sz, first, c, n, nbr, cnt, v, v_out, vin, resolve,
                                status, st);
        return;
    }
    auto walk = [&](auto k) {
        launch_k_smem(k, blocks_for(n, bs), bs, queue_bytes(bs), st, xs, sx, sy, sz, first, c, n,
                      nbr, cnt, v, v_out, vin, resolve, status);
    };
    const bool b = c.scenes != nullptr;
    if (c.nb_off) {
        walk(b ? k_search_xsph<true, true> : k_search_xsph<false, true>);
        launch_count_and_scan(xs, sx, sy, sz, first, c, n, cnt, status, st);
    }
    walk(b ? k_search_xsph<true, false> : k_search_xsph<false, false>);
}

size_t nb_scan_scratch_words(size_t n) {
    const size_t tiles = (n + kScanTile - 1) / kScanTile;
    return 4 * (tiles + 1);  // 64-bit tile sums and totals, back to back and in slices
}

template <bool B>
void launch_delta_apply_b(const float4* xs, const uint32_t* nbr, const int* cnt, const float* lam,
                          const StepConst& c, int n, float4* xs_out, uint32_t* keys_out,
                          const CellBins& bins, uint8_t* moved, float4* pre, unsigned* status,
                          cudaStream_t st) {
    const int bs = tuned_block(c, n, kTunedDelta);
    if (const int L = group_lanes(c, n); L > 1) {
        launch_delta_group(L, bs, xs, nbr, cnt, lam, c, n, xs_out, keys_out, bins, moved, pre,
                           status, st);
        return;
    }
    auto run = [&](auto k) {
        launch_k(k, blocks_for(n, bs), bs, st, xs, nbr, cnt, lam, c, n, xs_out, keys_out, bins,
                 moved, pre, status);
    };
    switch (c.sc.k != 0.0f ? c.sc.n : 0) {
        case 1: run(k_delta_apply<1, B>); break;
        case 2: run(k_delta_apply<2, B>); break;
        case 3: run(k_delta_apply<3, B>); break;
        case 4: run(k_delta_apply<4, B>); break;
        default: run(k_delta_apply<0, B>); break;
    }
}
void launch_delta_apply(const float4* xs, const uint32_t* nbr, const int* cnt, const float* lam,
                        const StepConst& c, int n, float4* xs_out, uint32_t* keys_out,
                        const CellBins& bins, unsigned* status, cudaStream_t st, uint8_t* moved,
                        float4* pre) {
    if (c.scenes)
        launch_delta_apply_b<true>(xs, nbr, cnt, lam, c, n, xs_out, keys_out, bins, moved, pre,
                                   status, st);
    else
        launch_delta_apply_b<false>(xs, nbr, cnt, lam, c, n, xs_out, keys_out, bins, moved, pre,
                                    status, st);
}
void launch_finalize(const uint32_t* org, const float4* x_old, const float4* vin_old,
                     const float4* v_old, const uint32_t* id_old, const float4* xs, int n,
                     const StepConst& c, float4* v_new, float4* vin_new, uint32_t* id_new,
                     const unsigned* status, cudaStream_t st) {
    launch_k(k_finalize, blocks_for(n), kBlock, st, org, x_old, vin_old, v_old, id_old, xs, n, c,
             v_new, vin_new, id_new, status);
}
void launch_xsph(const float4* x, const float4* v, const uint32_t* nbr, const int* cnt,
                 const StepConst& c, int n, float4* v_out, const float4* vin, bool resolve,
                 const unsigned* status, cudaStream_t st) {
    const int bs = tuned_block(c, n, kTunedXsph);
    if (c.scenes)
        launch_k(k_xsph<true>, blocks_for(n, bs), bs, st, x, v, nbr, cnt, c, n, v_out, vin,
                 resolve, status);
    else
        launch_k(k_xsph<false>, blocks_for(n, bs), bs, st, x, v, nbr, cnt, c, n, v_out, vin,
                 resolve, status);
}
void launch_vorticity(const float4* x, const float4* v, const uint32_t* nbr, const int* cnt,
                      const StepConst& c, int n, float4* omega, bool store_norm,
                      const unsigned* status, cudaStream_t st) {
    const int bs = tuned_block(c, n, kTunedVorticity);
    if (const int L = group_lanes(c, n); L > 1) {
        launch_vorticity_group(L, bs, x, v, nbr, cnt, c, n, omega, store_norm, status, st);
        return;
    }
    launch_k(k_vorticity, blocks_for(n, bs), bs, st, x, v, nbr, cnt, c, n, omega, store_norm,
             status);
}
void launch_omega_norm(float4* omega, int n, cudaStream_t st) {
    launch_k(k_omega_norm, blocks_for(n), kBlock, st, omega, n);
}
void launch_confine(const float4* x, const uint32_t* nbr, const int* cnt, const float4* omega,
                    const float4* v, const StepConst& c, int n, float4* v_out,
                    const float4* vin, bool resolve, const unsigned* status, cudaStream_t st) {
    const int bs = tuned_block(c, n, kTunedConfine);
    if (const int L = group_lanes(c, n); L > 1) {
        launch_confine_group(L, bs, x, nbr, cnt, omega, v, c, n, v_out, vin, resolve, status, st);
        return;
    }
    if (c.scenes)
        launch_k(k_confine<true>, blocks_for(n, bs), bs, st, x, nbr, cnt, omega, v, c, n, v_out,
                 vin, resolve, status);
    else
        launch_k(k_confine<false>, blocks_for(n, bs), bs, st, x, nbr, cnt, omega, v, c, n,
                 v_out, vin, resolve, status);
}
void launch_resolve(const float4* x, const float4* vin, float4* v, const StepConst& c, int n,
                    const unsigned* status, cudaStream_t st) {
    if (c.scenes)
        launch_k(k_resolve<true>, blocks_for(n), kBlock, st, x, vin, v, c, n, status);
    else
        launch_k(k_resolve<false>, blocks_for(n), kBlock, st, x, vin, v, c, n, status);
}
void launch_scatter_by_id(const float4* vals, const uint32_t* id, float4* out, int n,
                          cudaStream_t st) {
    k_scatter_by_id<<<blocks_for(n), kBlock, 0, st>>>(vals, id, out, n);
}
void launch_iota(uint32_t* a, int n, cudaStream_t st) {
    k_iota<<<blocks_for(n), kBlock, 0, st>>>(a, n);
}
void launch_density(const float4* x, const uint32_t* nbr, const int* cnt, const StepConst& c,
                    int n, size_t slots, float* err, cudaStream_t st) {
    k_density<<<blocks_for(n), kBlock, 0, st>>>(x, nbr, cnt, c, n, static_cast<uint32_t>(slots),
                                                err);
}
void launch_grid_keys(const float4* pos, uint32_t* keys, int n, const GridConst& g,
                      cudaStream_t st) {
    k_grid_keys<<<blocks_for(n), kBlock, 0, st>>>(pos, keys, n, g);
}
void launch_lambda_list(const float4* xs, const uint32_t* nbr, const int* cnt,
                        const StepConst& c, int n, float* lam, cudaStream_t st) {
    k_lambda_list<<<blocks_for(n), kBlock, 0, st>>>(xs, nbr, cnt, c, n, lam);
}
void launch_delta_list(const float4* xs, const uint32_t* nbr, const int* cnt, const float* lam,
                       const StepConst& c, int n, float4* delta, cudaStream_t st) {
    k_delta_list<<<blocks_for(n), kBlock, 0, st>>>(xs, nbr, cnt, lam, c, n, delta);
}
void launch_collide(float4* pos, int n, const StepConst& c, int kind, unsigned* flag,
                    cudaStream_t st) {
    k_collide<<<blocks_for(n), kBlock, 0, st>>>(pos, n, c, kind, flag);
}
void launch_integrate(const float4* x, float4* xs, float4* v, int n, const StepConst& c,
                      cudaStream_t st) {
    k_integrate<<<blocks_for(n), kBlock, 0, st>>>(x, xs, v, n, c);
}

}  // namespace pbf
