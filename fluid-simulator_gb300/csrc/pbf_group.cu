// pbf_group.cu -- the neighbour kernels with a group of lanes per particle, for
// scenes too small to fill the GPU with one thread per particle, where a
// launch takes as long as one thread's serial chain: nine rows of candidates,
// then list entry, gather and some 40 dependent operations per neighbour (some
// 5,700 instructions of the one-lane walk at about 8 cycles each when a
// scheduler has one warp: 25 us whatever the size).
//
// The group shares every part of that chain: the walk's rows go to nine lanes,
// and the neighbours' terms are formed side by side and left in a stash in
// shared memory.  The sums alone are serial: each lane adds the stashed terms
// in list order, the one-lane operations in the one-lane order, so lists and
// sums are the one-lane kernels', entry for entry and bit for bit.
//
// Measured on a GB300 against the lane groups these replace (8 lanes sharing
// each chunk of candidates, terms handed to lane 0 by shuffles): step of
// 1,024 particles 128 -> 88 us of kernels, 11,339 (3 iterations) 122 -> 104,
// 16,384 195 -> 177.
#include "pbf_device.cuh"

#include "pbf_common.h"

namespace pbf {
namespace {

// Stash entries (float4) per warp; a group has 8 L of them, and a longer list
// takes several rounds.
constexpr int kStash = 256;

// A particle's list shared by L lanes.
template <int L>
struct Group {
    static constexpr int kCap = kStash * L / 32;  // stash entries of a group
    int i, sub;
    unsigned mask;
    float4* stash;

    // The calling thread's particle and lane; false for threads past the last
    // particle (whole groups) and, group-wide, once a fatal status bit is set.
    __device__ __forceinline__ bool init(int n, const unsigned* status) {
        extern __shared__ float4 group_smem[];
        const int t = blockIdx.x * blockDim.x + threadIdx.x;
        i = t / L;
        sub = t % L;
        stash = group_smem + static_cast<size_t>(threadIdx.x / L) * kCap;
        if (i >= n) return false;
        const unsigned lane = threadIdx.x & 31u;
        mask = L == 32 ? 0xffffffffu : ((1u << (L % 32)) - 1u) << (lane & ~(L - 1u));
        return !__any_sync(mask, fatal(status));
    }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }

    // A sum over a list of count entries: term(j) is evaluated by the lanes
    // side by side, add(term) by every lane in list order.
    template <class Term, class Add>
    __device__ __forceinline__ void sum_list(const uint32_t* __restrict__ row, size_t st, int count,
                                             Term term, Add add) {
        for (int k0 = 0; k0 < count; k0 += kCap) {
            const int m = min(kCap, count - k0);
            sync();
            // Two entries a lane at a time: their loads overlap.
            for (int k = sub; k < m; k += 2 * L) {
                const bool two = k + L < m;
                const uint32_t ja = __ldg(&row[static_cast<size_t>(k0 + k) * st]);
                const uint32_t jb = two ? __ldg(&row[static_cast<size_t>(k0 + k + L) * st]) : ja;
                const float4 ta = term(ja), tb = term(jb);
                stash[k] = ta;
                if (two) stash[k + L] = tb;
            }
            sync();
#pragma unroll 4
            for (int k = 0; k < m; ++k) add(stash[k]);
        }
    }
};

// ---------------------------------------------------------------------------
// The walk: nine lanes per particle, one stencil row each, three particles a
// warp.  A lane tests its row's candidates 32 at a time into hit masks, the
// group scans the rows' counts (the list's order is row after row), and each
// lane writes its hits at their places: into the list and, up to kRowCap, into
// the particle's stash, where the lanes then form the neighbours' terms.
// Nine rows side by side instead of one after the other: a launch is as long
// as one row, and a lane does one ninth of the one-lane work (with 8, 16 or 32
// lanes on the same row instead, the places of each chunk's hits cost more
// than its tests).
// ---------------------------------------------------------------------------
constexpr int kRowLanes = 9, kRowParts = 3;
constexpr int kRowCap = 64;                // stash entries per particle
constexpr int kRowStride = kRowCap + 1;    // 16 bytes apart in the banks

struct RowGroup {
    int i, sub, base;  // particle (clamped), row, first lane of the group
    bool valid;        // lanes of a particle
    float4* stash;

    // The calling thread's particle and row; false for whole warps past the
    // last particle and, warp-wide, once a fatal status bit is set.
    __device__ __forceinline__ bool init(int n, const unsigned* status) {
        extern __shared__ float4 row_smem[];
        const int lane = threadIdx.x & 31;
        const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
        const int g = lane / kRowLanes;
        if (warp * kRowParts >= n) return false;
        i = warp * kRowParts + g;
        base = g * kRowLanes;
        sub = lane - base;
        valid = g < kRowParts && i < n;
        i = min(i, n - 1);
        stash = row_smem + ((threadIdx.x >> 5) * kRowParts + min(g, kRowParts - 1)) * kRowStride;
        return !__any_sync(0xffffffffu, fatal(status));
    }
};

// Hit bits of 32 candidates of the row range [s, e) from j (a multiple of 4;
// candidate j is the highest bit), less the particle itself; 8 at a time, as
// far as the range goes (16 at a time: 1.4 % more of a step of 16,384 particles).
// h2u: the float above h2 (d2 <= h2 exactly when d2 - h2u has its sign set).
__device__ __forceinline__ uint32_t row_hits(float4 pi, float h2u, const float* __restrict__ sx,
                                             const float* __restrict__ sy,
                                             const float* __restrict__ sz, int j, int s, int e,
                                             int self) {
    uint32_t acc = 0u;
#pragma unroll 1
    for (int t = j; t < j + 32; t += 8) {
        if (t >= e) {
            acc <<= j + 32 - t;
            break;
        }
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
            const float4 X = __ldg(reinterpret_cast<const float4*>(sx + t + q));
            const float4 Y = __ldg(reinterpret_cast<const float4*>(sy + t + q));
            const float4 Z = __ldg(reinterpret_cast<const float4*>(sz + t + q));
            const float x[4] = {X.x, X.y, X.z, X.w}, y[4] = {Y.x, Y.y, Y.z, Y.w},
                        z[4] = {Z.x, Z.y, Z.z, Z.w};
#pragma unroll
            for (int k = 0; k < 4; ++k)
                acc = __funnelshift_l(
                    __float_as_uint(fsub(
                        dist2(fsub(pi.x, x[k]), fsub(pi.y, y[k]), fsub(pi.z, z[k])), h2u)),
                    acc, 1);
        }
    }
    const uint32_t past = __funnelshift_rc(0xffffffffu, 0u, e - j);
    const uint32_t me = __funnelshift_rc(0x80000000u, 0u, static_cast<uint32_t>(self - j));
    return acc & (0xffffffffu >> max(s - j, 0)) & ~(past | me);
}

// The walk of the warp's particles (slot-major or compact list at out, at
// most c.max_nb entries, the first kRowCap also in the stash as bits of j);
// returns the count on every lane of the group.  Radius 1.
template <bool B>
__device__ __forceinline__ int row_walk(const RowGroup& gr, const StepConst& c, float4 pi,
                                        const float* __restrict__ sx, const float* __restrict__ sy,
                                        const float* __restrict__ sz,
                                        const int* __restrict__ first,
                                        uint32_t* __restrict__ out) {
    int s = 0, e = 0;
    {
        const StencilRows<B> rows(c, gr.i, pi);
        const int z = rows.cz - 1 + gr.sub / 3, y = rows.cy - 1 + gr.sub % 3;
        if (gr.valid && z >= rows.z0 && z <= rows.z1 && y >= rows.y0 && y <= rows.y1 &&
            !rows.range(first, z, y, s, e))
            s = e = 0;
    }
    const float h2u = __uint_as_float(__float_as_uint(c.k.h2) + 1u);
    const int a = s & ~3;
    uint32_t m0 = 0u, m1 = 0u;
    int place = 0;
    if (s < e) {
        m0 = row_hits(pi, h2u, sx, sy, sz, a, s, e, gr.i);
        if (a + 32 < e) m1 = row_hits(pi, h2u, sx, sy, sz, a + 32, s, e, gr.i);
        place = __popc(m0) + __popc(m1);
        for (int j = a + 64; j < e; j += 32)
            place += __popc(row_hits(pi, h2u, sx, sy, sz, j, s, e, gr.i));
    }
    const int mine = place;
#pragma unroll
    for (int o = 1; o < kRowLanes; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, place, o);
        if (gr.sub >= o) place += t;
    }
    const int count = __shfl_sync(0xffffffffu, place, gr.base + kRowLanes - 1);
    place -= mine;
    const size_t stride = nb_step(c);
    uint32_t* dst = out + static_cast<size_t>(place) * stride;
    for (int j = a; j < e; j += 32) {
        uint32_t m = j == a ? m0 : m1;
        if (j > a + 32) m = row_hits(pi, h2u, sx, sy, sz, j, s, e, gr.i);
        while (m) {
            const int b = 31 - __clz(m);
            m ^= 1u << b;
            const int k = j + 31 - b;
            if (place < c.max_nb) *dst = static_cast<uint32_t>(k);
            if (place < kRowCap) gr.stash[place].x = __int_as_float(k);
            dst += stride;
            ++place;
        }
    }
    return count;
}

// Sums over the group's list (count entries, as row_walk left them): term(j)
// by the lanes side by side, add(term) by every lane in list order.
template <class Term, class Add>
__device__ __forceinline__ void row_sum(const RowGroup& gr, int count,
                                        const uint32_t* __restrict__ out, size_t stride, Term term,
                                        Add add) {
    for (int k0 = 0; __any_sync(0xffffffffu, k0 < count); k0 += kRowCap) {
        const int m = max(0, min(kRowCap, count - k0));
        __syncwarp();
        for (int k = gr.sub; k < m; k += kRowLanes) {
            const int j = k0 == 0 ? __float_as_int(gr.stash[k].x)
                                  : static_cast<int>(out[static_cast<size_t>(k0 + k) * stride]);
            gr.stash[k] = term(j);
        }
        __syncwarp();
#pragma unroll 4
        for (int k = 0; k < m; ++k) add(gr.stash[k]);
    }
}

// k_search (walk, optional lambda).
template <bool LAMBDA, bool B>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_search_rows(const float4* __restrict__ xs, const float* __restrict__ sx,
              const float* __restrict__ sy, const float* __restrict__ sz,
              const int* __restrict__ first, StepConst c, int n, uint32_t* __restrict__ nbr,
              int* __restrict__ cnt, float* __restrict__ lam, unsigned* __restrict__ status) {
    RowGroup gr;
    if (!gr.init(n, status)) return;
    const int i = gr.i;
    const float4 pi = xs[i];
    uint32_t* __restrict__ out = nbr + nb_first(c, i);
    const int count = row_walk<B>(gr, c, pi, sx, sy, sz, first, out);
    LambdaAcc acc{c.k.c_poly6, 0.0f, 0.0f, 0.0f, 0.0f};
    if constexpr (LAMBDA)
        row_sum(
            gr, gr.valid && count <= c.max_nb ? count : 0, out, nb_step(c),
            [&](int j) {
                const float4 pj = __ldg(&xs[j]);
                const float dx = fsub(pi.x, pj.x), dy = fsub(pi.y, pj.y), dz = fsub(pi.z, pj.z);
                const float d2 = dist2(dx, dy, dz);
                float4 t;
                spiky(c.k, dx, dy, dz, d2, t.x, t.y, t.z);
                t.w = poly6(c.k, d2);
                return t;
            },
            [&](float4 t) {
                acc.wsum = fadd(acc.wsum, t.w);
                acc.s2 = ffma(t.z, t.z, ffma(t.y, t.y, ffma(t.x, t.x, acc.s2)));
                acc.gx = fadd(acc.gx, t.x);
                acc.gy = fadd(acc.gy, t.y);
                acc.gz = fadd(acc.gz, t.z);
            });
    if (!gr.valid || gr.sub != 0) return;
    cnt[i] = count;
    if (count > c.max_nb) atomicOr(status, kStatusNeighborOverflow);
    if (LAMBDA) lam[i] = count > c.max_nb ? CUDART_NAN_F : lambda_of_acc<B>(c, i, acc);
}

// k_search_xsph (final walk, XSPH, optional velocity response).
template <bool B>
__global__ void __maxnreg__(56)  // 36 warps an SM: 16,384 particles in one wave
k_search_xsph_rows(const float4* __restrict__ xs, const float* __restrict__ sx,
                   const float* __restrict__ sy, const float* __restrict__ sz,
                   const int* __restrict__ first, StepConst c, int n, uint32_t* __restrict__ nbr,
                   int* __restrict__ cnt, const float4* __restrict__ v, float4* __restrict__ v_out,
                   const float4* __restrict__ vin, bool resolve, unsigned* __restrict__ status) {
    RowGroup gr;
    if (!gr.init(n, status)) return;
    const int i = gr.i;
    const float4 pi = xs[i], vi = v[i];
    uint32_t* __restrict__ out = nbr + nb_first(c, i);
    const int count = row_walk<B>(gr, c, pi, sx, sy, sz, first, out);
    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
    row_sum(
        gr, gr.valid && count <= c.max_nb ? count : 0, out, nb_step(c),
        [&](int j) {
            const float4 pj = __ldg(&xs[j]), vj = __ldg(&v[j]);
            return make_float4(
                fsub(vj.x, vi.x), fsub(vj.y, vi.y), fsub(vj.z, vi.z),
                poly6(c.k, dist2(fsub(pi.x, pj.x), fsub(pi.y, pj.y), fsub(pi.z, pj.z))));
        },
        [&](float4 t) {
            cx = ffma(t.x, t.w, cx);
            cy = ffma(t.y, t.w, cy);
            cz = ffma(t.z, t.w, cz);
        });
    if (!gr.valid || gr.sub != 0) return;
    cnt[i] = count;
    if (count > c.max_nb) atomicOr(status, kStatusNeighborOverflow);
    const float xc = B ? scene_of(c, i).xsph_c : c.xsph_c;
    float4 o = make_float4(ffma(xc, cx, vi.x), ffma(xc, cy, vi.y), ffma(xc, cz, vi.z), vi.w);
    if (!count_ok(count, c.max_nb))
        o = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, vi.w);
    if (resolve)
        resolve_velocity(colliders_of<B>(c, i), c.particle_radius, c.restitution, c.friction, pi,
                         vin[i], o);
    v_out[i] = o;
}

// scorr with the exponent read at run time, the common ones unrolled (the
// products are the same).
__device__ __forceinline__ float scorr_n(const ScorrConst& s, float d2) {
    switch (s.n) {
        case 1: return scorr<1>(s, d2);
        case 2: return scorr<2>(s, d2);
        case 3: return scorr<3>(s, d2);
        case 4: return scorr<4>(s, d2);
        default: return scorr<0>(s, d2);
    }
}

// k_delta_apply (delta p, collision projection, next keys).
template <bool B, int L>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_delta_group(const float4* __restrict__ xs, const uint32_t* __restrict__ nbr,
              const int* __restrict__ cnt, const float* __restrict__ lam, StepConst c, int n,
              float4* __restrict__ xs_out, uint32_t* __restrict__ keys_out, CellBins bins,
              uint8_t* __restrict__ moved, float4* __restrict__ pre,
              unsigned* __restrict__ status) {
    Group<L> gr;
    if (!gr.init(n, status)) return;
    const int i = gr.i;
    const float4 pi = xs[i];
    const int count = cnt[i];
    const float li = lam[i];
    float dpx, dpy, dpz;
    if (!count_ok(count, c.max_nb)) {
        dpx = dpy = dpz = CUDART_NAN_F;
    } else {
        float ax = 0.0f, ay = 0.0f, az = 0.0f;
        gr.sum_list(
            nbr + nb_first(c, i), nb_step(c), count,
            [&](uint32_t j) {
                const float4 pj = __ldg(&xs[j]);
                const float lj = __ldg(&lam[j]);
                const float dx = fsub(pi.x, pj.x), dy = fsub(pi.y, pj.y), dz = fsub(pi.z, pj.z);
                const float d2 = dist2(dx, dy, dz);
                float4 t;
                spiky(c.k, dx, dy, dz, d2, t.x, t.y, t.z);
                t.w = fadd(fadd(li, lj), scorr_n(c.sc, d2));
                return t;
            },
            [&](float4 t) {
                ax = ffma(t.w, t.x, ax);
                ay = ffma(t.w, t.y, ay);
                az = ffma(t.w, t.z, az);
            });
        const float gs = B ? scene_of(c, i).gs : c.gs;
        dpx = fmul(gs, ax);
        dpy = fmul(gs, ay);
        dpz = fmul(gs, az);
    }
    if (gr.sub == 0)
        apply_delta<B>(c, i, pi, dpx, dpy, dpz, xs_out, keys_out, bins, moved, pre, status);
}

// k_vorticity.
template <int L>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_vorticity_group(const float4* __restrict__ x, const float4* __restrict__ v,
                  const uint32_t* __restrict__ nbr, const int* __restrict__ cnt, StepConst c,
                  int n, float4* __restrict__ omega, bool store_norm,
                  const unsigned* __restrict__ status) {
    Group<L> gr;
    if (!gr.init(n, status)) return;
    const int i = gr.i;
    const int count = cnt[i];
    if (!count_ok(count, c.max_nb)) {
        if (gr.sub == 0)
            omega[i] = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F,
                                   store_norm ? CUDART_NAN_F : 0.0f);
        return;
    }
    const float4 pi = x[i], vi = v[i];
    float ox = 0.0f, oy = 0.0f, oz = 0.0f;
    gr.sum_list(
        nbr + nb_first(c, i), nb_step(c), count,
        [&](uint32_t j) {
            const float4 pj = __ldg(&x[j]), vj = __ldg(&v[j]);
            const float dx = fsub(pi.x, pj.x), dy = fsub(pi.y, pj.y), dz = fsub(pi.z, pj.z);
            float gx, gy, gz;
            spiky(c.k, dx, dy, dz, dist2(dx, dy, dz), gx, gy, gz);
            const float vx = fsub(vj.x, vi.x), vy = fsub(vj.y, vi.y), vz = fsub(vj.z, vi.z);
            return make_float4(crossc(gy, gz, vy, vz), crossc(gz, gx, vz, vx),
                               crossc(gx, gy, vx, vy), 0.0f);
        },
        [&](float4 t) {
            ox = fadd(ox, t.x);
            oy = fadd(oy, t.y);
            oz = fadd(oz, t.z);
        });
    if (gr.sub == 0) omega[i] = make_float4(ox, oy, oz, store_norm ? len3(ox, oy, oz) : 0.0f);
}

// k_confine (confinement, optional velocity response).
template <bool B, int L>
__global__ void __launch_bounds__(kMaxTunedBlock)
k_confine_group(const float4* __restrict__ x, const uint32_t* __restrict__ nbr,
                const int* __restrict__ cnt, const float4* __restrict__ om,
                const float4* __restrict__ v, StepConst c, int n, float4* __restrict__ v_out,
                const float4* __restrict__ vin, bool resolve,
                const unsigned* __restrict__ status) {
    Group<L> gr;
    if (!gr.init(n, status)) return;
    const int i = gr.i;
    const int count = cnt[i];
    const float4 pi = x[i], vi = v[i], wi = om[i];
    float4 o = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, vi.w);
    if (count_ok(count, c.max_nb)) {
        float ex = 0.0f, ey = 0.0f, ez = 0.0f;
        gr.sum_list(
            nbr + nb_first(c, i), nb_step(c), count,
            [&](uint32_t j) {
                const float4 pj = __ldg(&x[j]);
                const float wj = __ldg(&om[j].w);
                const float dx = fsub(pi.x, pj.x), dy = fsub(pi.y, pj.y), dz = fsub(pi.z, pj.z);
                float4 t;
                spiky(c.k, dx, dy, dz, dist2(dx, dy, dz), t.x, t.y, t.z);
                t.w = fsub(wj, wi.w);
                return t;
            },
            [&](float4 t) {
                ex = ffma(t.w, t.x, ex);
                ey = ffma(t.w, t.y, ey);
                ez = ffma(t.w, t.z, ez);
            });
        o = confine_finish(c, ex, ey, ez, wi, vi);
    }
    if (gr.sub != 0) return;
    if (resolve)
        resolve_velocity(colliders_of<B>(c, i), c.particle_radius, c.restitution, c.friction, pi,
                         vin[i], o);
    v_out[i] = o;
}

size_t stash_bytes(int block) { return sizeof(float4) * kStash * static_cast<size_t>(block / 32); }

int row_particles(int block) { return block / 32 * kRowParts; }
size_t row_bytes(int block) {
    return sizeof(float4) * kRowStride * static_cast<size_t>(row_particles(block));
}

// Calls f(integral_constant of the group size) for L in {2, 4, 8, 16, 32}.
template <class F>
void with_lanes(int L, F f) {
    switch (L) {
        case 32: f(std::integral_constant<int, 32>()); break;
        case 16: f(std::integral_constant<int, 16>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        default: f(std::integral_constant<int, 2>()); break;
    }
}

}  // namespace

void launch_search_rows(int bs, const float4* xs, const float* sx, const float* sy,
                        const float* sz, const int* first, const StepConst& c, int n,
                        uint32_t* nbr, int* cnt, float* lam, unsigned* status, bool with_lambda,
                        cudaStream_t st) {
    auto k = with_lambda ? (c.scenes ? k_search_rows<true, true> : k_search_rows<true, false>)
                         : (c.scenes ? k_search_rows<false, true> : k_search_rows<false, false>);
    launch_k_smem(k, blocks_for(n, row_particles(bs)), bs, row_bytes(bs), st, xs, sx, sy, sz,
                  first, c, n, nbr, cnt, lam, status);
}

void launch_search_xsph_rows(int bs, const float4* xs, const float* sx, const float* sy,
                             const float* sz, const int* first, const StepConst& c, int n,
                             uint32_t* nbr, int* cnt, const float4* v, float4* v_out,
                             const float4* vin, bool resolve, unsigned* status, cudaStream_t st) {
    launch_k_smem(c.scenes ? k_search_xsph_rows<true> : k_search_xsph_rows<false>,
                  blocks_for(n, row_particles(bs)), bs, row_bytes(bs), st, xs, sx, sy, sz, first,
                  c, n, nbr, cnt, v, v_out, vin, resolve, status);
}

void launch_delta_group(int L, int bs, const float4* xs, const uint32_t* nbr, const int* cnt,
                        const float* lam, const StepConst& c, int n, float4* xs_out,
                        uint32_t* keys_out, const CellBins& bins, uint8_t* moved, float4* pre,
                        unsigned* status, cudaStream_t st) {
    with_lanes(L, [&](auto l) {
        constexpr int K = decltype(l)::value;
        launch_k_smem(c.scenes ? k_delta_group<true, K> : k_delta_group<false, K>,
                      blocks_for(static_cast<size_t>(n) * K, bs), bs, stash_bytes(bs), st, xs, nbr,
                      cnt, lam, c, n, xs_out, keys_out, bins, moved, pre, status);
    });
}

void launch_vorticity_group(int L, int bs, const float4* x, const float4* v, const uint32_t* nbr,
                            const int* cnt, const StepConst& c, int n, float4* omega,
                            bool store_norm, const unsigned* status, cudaStream_t st) {
    with_lanes(L, [&](auto l) {
        constexpr int K = decltype(l)::value;
        launch_k_smem(k_vorticity_group<K>, blocks_for(static_cast<size_t>(n) * K, bs), bs,
                      stash_bytes(bs), st, x, v, nbr, cnt, c, n, omega, store_norm, status);
    });
}

void launch_confine_group(int L, int bs, const float4* x, const uint32_t* nbr, const int* cnt,
                          const float4* omega, const float4* v, const StepConst& c, int n,
                          float4* v_out, const float4* vin, bool resolve, const unsigned* status,
                          cudaStream_t st) {
    with_lanes(L, [&](auto l) {
        constexpr int K = decltype(l)::value;
        launch_k_smem(c.scenes ? k_confine_group<true, K> : k_confine_group<false, K>,
                      blocks_for(static_cast<size_t>(n) * K, bs), bs, stash_bytes(bs), st, x, nbr,
                      cnt, omega, v, c, n, v_out, vin, resolve, status);
    });
}

}  // namespace pbf
