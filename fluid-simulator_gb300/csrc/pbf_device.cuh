// pbf_device.cuh -- device helpers shared by the step's kernels (pbf_kernels.cu:
// one thread per particle; pbf_group.cu: a group of lanes per particle).
#pragma once

#include <math_constants.h>

#include "pbf_kernels.cuh"

namespace pbf {
namespace {

__device__ __forceinline__ bool fatal(const unsigned* status) {
    return status != nullptr && (__ldcg(status) & kStatusFatalMask) != 0u;
}

// The scene of particle slot i in a batched solver.
__device__ __forceinline__ const SceneConst& scene_of(const StepConst& c, int i) {
    return c.scenes[__ldg(&c.sid[i])];
}

// First entry and entry stride of particle i's neighbour list.
__device__ __forceinline__ size_t nb_first(const StepConst& c, int i) {
    return c.nb_off ? static_cast<size_t>(__ldg(&c.nb_off[i])) : static_cast<size_t>(i);
}
__device__ __forceinline__ size_t nb_step(const StepConst& c) {
    return c.nb_off ? static_cast<size_t>(__ldg(c.nb_step)) : c.stride;
}

// Grid and first global cell key of slot i: the scene's (B) or c.g.
template <bool B>
__device__ __forceinline__ void grid_of(const StepConst& c, int i, GridConst& g, uint32_t& base) {
    if constexpr (B) {
        const SceneConst& s = scene_of(c, i);
        g = s.g;
        base = s.cell_base;
    } else {
        g = c.g;
        base = 0u;
    }
}

// Colliders with the container of slot i's scene (B) or c.col.
template <bool B>
__device__ __forceinline__ Colliders colliders_of(const StepConst& c, int i) {
    Colliders col = c.col;
    if constexpr (B) {
        const SceneConst& s = scene_of(c, i);
        col.cminx = s.cminx;
        col.cminy = s.cminy;
        col.cminz = s.cminz;
        col.cmaxx = s.cmaxx;
        col.cmaxy = s.cmaxy;
        col.cmaxz = s.cmaxz;
    }
    return col;
}

// The key of particle i for the next rebuild, counted in its cell.
__device__ __forceinline__ void put_key(uint32_t* __restrict__ keys, const CellBins& bins, int i,
                                        uint32_t key) {
    keys[i] = key;
    if (bins.count) bins.place[i] = atomicAdd(&bins.count[key], 1u);
    if (bins.sums) count_tile(bins.sums, bins.shift, key);
}

// Accumulated constraint terms of computeLambda (pbf_solver_kernels.cu:26-105).
struct LambdaAcc {
    float wsum, s2, gx, gy, gz;
};

__device__ __forceinline__ void lambda_add(const KernelConst& k, LambdaAcc& a, float dx, float dy,
                                           float dz, float d2) {
    a.wsum = fadd(a.wsum, poly6(k, d2));
    float gx, gy, gz;
    spiky(k, dx, dy, dz, d2, gx, gy, gz);
    a.s2 = ffma(gz, gz, ffma(gy, gy, ffma(gx, gx, a.s2)));
    a.gx = fadd(a.gx, gx);
    a.gy = fadd(a.gy, gy);
    a.gz = fadd(a.gz, gz);
}

__device__ __forceinline__ float lambda_finish(float mass, float rho0, float gs2, float eps,
                                               const LambdaAcc& a) {
    const float rho = fmul(mass, a.wsum);
    const float g2 = dist2(a.gx, a.gy, a.gz);
    const float denom = ffma(gs2, fadd(a.s2, g2), eps);
    const float C = fsub(fdiv(rho, rho0), 1.0f);
    return fdiv(-C, denom);
}
__device__ __forceinline__ float lambda_finish(const StepConst& c, const LambdaAcc& a) {
    return lambda_finish(c.mass, c.rho0, c.gs2, c.lambda_eps, a);
}

template <bool B>
__device__ __forceinline__ float lambda_of_acc(const StepConst& c, int i, const LambdaAcc& acc) {
    if constexpr (B) {
        const SceneConst& sc = scene_of(c, i);
        return lambda_finish(sc.mass, sc.rho0, sc.gs2, c.lambda_eps, acc);
    } else {
        return lambda_finish(c, acc);
    }
}

// Squared distances from coordinate p to the slabs of the cells below and
// above cell k on one axis (cell k spans [lo + k cell, lo + (k + 1) cell);
// the clamped end cells extend to infinity, which changes neither distance),
// each first reduced by eps.  Margin arithmetic only: it decides which cells
// the walk reads, never a neighbour.
__device__ __forceinline__ void slab_dist2(float p, float lo, float cell, int k, float eps,
                                           float& below, float& above) {
    const float b0 = fmaf(static_cast<float>(k), cell, lo);
    const float b1 = fmaf(static_cast<float>(k + 1), cell, lo);
    const float d0 = fmaxf(p - b0 - eps, 0.0f);
    const float d1 = fmaxf(b1 - p - eps, 0.0f);
    below = d0 * d0;
    above = d1 * d1;
}

// The stencil rows of particle i, as the walks visit them: z0..z1 x y0..y1
// (clamped to the grid), and range(z, y) gives row (z, y)'s candidate index
// range [s, e): its cells x0..x1 are consecutive keys.  Keys fit in 32 bits
// (cells < 2^32 is checked at initialisation), so the reference's 64-bit key
// arithmetic truncates to the same values.
// Cell pruning (radius 1): a stencil cell whose box lies farther than h
// from the particle holds no neighbour, so range() returns false for the
// rows (y, z) that far and leaves out the end cells of a row that far.  Per
// axis, eps = 2^-14 (|p| + |min| + cell) covers the FP32 rounding of every
// cell index (floor((p - min) / cell)) and of the candidates' differences,
// and the bound h2 (1 + 2^-10) the rounding of d2: only certain misses are
// left out, so the list is entry for entry the unpruned walk's.
template <bool B>
struct StencilRows {
    GridConst g;
    uint32_t base, gx, gxy;
    int cx, cy, cz, x0, x1, y0, y1, z0, z1;
    bool prune;
    float xb2, xa2, yb2, ya2, zb2, za2, lim2;
    __device__ __forceinline__ StencilRows(const StepConst& c, int i, float4 pi) {
        grid_of<B>(c, i, g, base);
        cell_of(g, pi.x, pi.y, pi.z, cx, cy, cz);
        const int R = g.radius;
        x0 = max(0, cx - R);
        x1 = min(g.gx - 1, cx + R);
        y0 = max(0, cy - R);
        y1 = min(g.gy - 1, cy + R);
        z0 = max(0, cz - R);
        z1 = min(g.gz - 1, cz + R);
        gx = static_cast<uint32_t>(g.gx);
        gxy = gx * static_cast<uint32_t>(g.gy);
        prune = c.prune_cells && R == 1;
        xb2 = xa2 = yb2 = ya2 = zb2 = za2 = lim2 = 0.0f;
        if (prune) {
            const float eps = 6.103515625e-05f *
                              (fabsf(pi.x) + fabsf(pi.y) + fabsf(pi.z) + fabsf(g.minx) +
                               fabsf(g.miny) + fabsf(g.minz) + g.cell);
            slab_dist2(pi.x, g.minx, g.cell, cx, eps, xb2, xa2);
            slab_dist2(pi.y, g.miny, g.cell, cy, eps, yb2, ya2);
            slab_dist2(pi.z, g.minz, g.cell, cz, eps, zb2, za2);
            lim2 = c.k.h2 * 1.0009765625f;
        }
    }
    __device__ __forceinline__ bool range(const int* __restrict__ first, int z, int y, int& s,
                                          int& e) const {
        int xa = x0, xb = x1;
        if (prune) {
            const float dyz = (z < cz ? zb2 : (z > cz ? za2 : 0.0f)) +
                              (y < cy ? yb2 : (y > cy ? ya2 : 0.0f));
            if (dyz > lim2) return false;
            if (xa < cx && dyz + xb2 > lim2) xa = cx;
            if (xb > cx && dyz + xa2 > lim2) xb = cx;
        }
        const uint32_t row =
            base + static_cast<uint32_t>(y) * gx + static_cast<uint32_t>(z) * gxy;
        s = __ldg(&first[row + static_cast<uint32_t>(xa)]);
        e = __ldg(&first[row + static_cast<uint32_t>(xb) + 1u]);
        return true;
    }
};

__device__ __forceinline__ bool count_ok(int count, int max_nb) {
    return count >= 0 && count <= max_nb;
}

// What k_delta_apply does once particle i's delta p is known: the move, the
// collision projection and the key.  moved (optional): bit a set where the
// projection changed component a.  pre (optional): the position before the
// projection.
template <bool B>
__device__ __forceinline__ void apply_delta(const StepConst& c, int i, float4 pi, float dpx,
                                            float dpy, float dpz, float4* __restrict__ xs_out,
                                            uint32_t* __restrict__ keys_out, const CellBins& bins,
                                            uint8_t* __restrict__ moved, float4* __restrict__ pre,
                                            unsigned* __restrict__ status) {
    float px = fadd(pi.x, dpx), py = fadd(pi.y, dpy), pz = fadd(pi.z, dpz);
    const float ux = px, uy = py, uz = pz;
    if (pre) pre[i] = make_float4(ux, uy, uz, pi.w);
    if (!project_all(colliders_of<B>(c, i), c.particle_radius, px, py, pz))
        atomicOr(status, kStatusNotConverged);
    if (moved)
        moved[i] = static_cast<uint8_t>((px != ux) | ((py != uy) << 1) | ((pz != uz) << 2));
    const float4 q = make_float4(px, py, pz, pi.w);
    xs_out[i] = q;
    if (keys_out) {
        GridConst g;
        uint32_t base;
        grid_of<B>(c, i, g, base);
        put_key(keys_out, bins, i, base + key_of(g, q));
    }
}

// The confinement velocity from the summed eta = sum (|w_j| - |w_i|) grad W.
__device__ __forceinline__ float4 confine_finish(const StepConst& c, float ex, float ey, float ez,
                                                 float4 wi, float4 vi) {
    const float el = len3(ex, ey, ez);
    float nx = 0.0f, ny = 0.0f, nz = 0.0f;
    if (el > kEtaEpsilon) {
        nx = fdiv(ex, el);
        ny = fdiv(ey, el);
        nz = fdiv(ez, el);
    }
    const float cx = fmul(c.vort_eps, crossc(ny, nz, wi.y, wi.z));
    const float cy = fmul(c.vort_eps, crossc(nz, nx, wi.z, wi.x));
    const float cz = fmul(c.vort_eps, crossc(nx, ny, wi.x, wi.y));
    return make_float4(ffma(c.dt, cx, vi.x), ffma(c.dt, cy, vi.y), ffma(c.dt, cz, vi.z), vi.w);
}

}  // namespace
}  // namespace pbf
