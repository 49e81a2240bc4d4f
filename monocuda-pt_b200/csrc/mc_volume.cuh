// mc_volume.cuh - heterogeneous media: the dense density grid, its trilinear
// sample, and the two trackers of PT:784-838.
//
// The reference reads a NanoVDB FloatGrid (PT:784-789: worldToIndexF, then
// nanovdb::math::createSampler<1>, a trilinear sampler with background 0).
// mc_volume_grid is a dense stand-in with the same reading: index point
// (p - origin) * inv_voxel_size, the 8 voxels around its floor, interpolated
// along z, then y, then x. Delta tracking (free flight) and ratio tracking
// (transmittance) follow PT:796-815 and PT:817-838 step for step, so that
// they draw the same random numbers in the same order as the reference.
#pragma once

#include "mc_math.cuh"

namespace mc {

constexpr int kVolumeHeaderBytes = 64;
static_assert(sizeof(mc_volume_grid) == kVolumeHeaderBytes, "the voxels follow the 64-byte header");

MC_D const float* volume_voxels(const mc_volume_grid* g) {
    return reinterpret_cast<const float*>(reinterpret_cast<const char*>(g) + kVolumeHeaderBytes);
}

MC_D float volume_lerp(float a, float b, float w) { return fmaf(w, b - a, a); }

// Grid value at world point p (0 outside the voxels).
MC_D float volume_density(const mc_volume_grid* g, const V3& p) {
    const float inv = g->inv_voxel_size;
    const float x = (p.x - g->origin[0]) * inv;
    const float y = (p.y - g->origin[1]) * inv;
    const float z = (p.z - g->origin[2]) * inv;
    const int nx = g->dims[0], ny = g->dims[1], nz = g->dims[2];
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    // all 8 voxels outside (or a NaN coordinate): every term is 0
    if (!(fx >= -1.0f && fx <= (float)(nx - 1) && fy >= -1.0f && fy <= (float)(ny - 1) && fz >= -1.0f &&
          fz <= (float)(nz - 1)))
        return 0.0f;
    const int i = (int)fx, j = (int)fy, k = (int)fz;
    const float u = x - fx, v = y - fy, w = z - fz;
    const float* vox = volume_voxels(g);
    auto at = [&](int a, int b, int c) -> float {
        if (a < 0 || b < 0 || c < 0 || a >= nx || b >= ny || c >= nz) return 0.0f;
        return __ldg(vox + a + (long long)nx * (b + (long long)ny * c));
    };
    const float c00 = volume_lerp(at(i, j, k), at(i, j, k + 1), w);
    const float c01 = volume_lerp(at(i, j + 1, k), at(i, j + 1, k + 1), w);
    const float c10 = volume_lerp(at(i + 1, j, k), at(i + 1, j, k + 1), w);
    const float c11 = volume_lerp(at(i + 1, j + 1, k), at(i + 1, j + 1, k + 1), w);
    return volume_lerp(volume_lerp(c00, c01, v), volume_lerp(c10, c11, v), u);
}

// The densities at K distances along o + d t, all 8 K voxel reads in flight
// together: volume_density's values without its branches. Distances at or past
// `limit` are not read.
template <int K>
MC_D void volume_densities(const mc_volume_grid* g, const V3& o, const V3& d, const float* t, float limit, float* out) {
    const float inv = g->inv_voxel_size;
    const float gx = g->origin[0], gy = g->origin[1], gz = g->origin[2];
    const int nx = g->dims[0], ny = g->dims[1], nz = g->dims[2];
    const float* vox = volume_voxels(g);
    float c[K][8], w[K][3];
#pragma unroll
    for (int k = 0; k < K; k++) {
        const V3 p = o + d * t[k];
        const float x = (p.x - gx) * inv, y = (p.y - gy) * inv, z = (p.z - gz) * inv;
        const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
        const bool in = t[k] < limit && fx >= -1.0f && fx <= (float)(nx - 1) && fy >= -1.0f && fy <= (float)(ny - 1) &&
                        fz >= -1.0f && fz <= (float)(nz - 1);
        const int i = in ? (int)fx : 0, j = in ? (int)fy : 0, l = in ? (int)fz : 0;
        w[k][0] = x - fx;
        w[k][1] = y - fy;
        w[k][2] = z - fz;
        const bool x0 = in && i >= 0, x1 = in && i + 1 < nx, y0 = j >= 0, y1 = j + 1 < ny, z0 = l >= 0, z1 = l + 1 < nz;
        const float* v = vox + i + (long long)nx * (j + (long long)ny * l);
        const long long sy = nx, sz = (long long)nx * ny;
        c[k][0] = x0 && y0 && z0 ? __ldg(v) : 0.0f;
        c[k][1] = x0 && y0 && z1 ? __ldg(v + sz) : 0.0f;
        c[k][2] = x0 && y1 && z0 ? __ldg(v + sy) : 0.0f;
        c[k][3] = x0 && y1 && z1 ? __ldg(v + sy + sz) : 0.0f;
        c[k][4] = x1 && y0 && z0 ? __ldg(v + 1) : 0.0f;
        c[k][5] = x1 && y0 && z1 ? __ldg(v + 1 + sz) : 0.0f;
        c[k][6] = x1 && y1 && z0 ? __ldg(v + 1 + sy) : 0.0f;
        c[k][7] = x1 && y1 && z1 ? __ldg(v + 1 + sy + sz) : 0.0f;
        if (!in) w[k][0] = w[k][1] = w[k][2] = 0.0f;
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        const float c00 = volume_lerp(c[k][0], c[k][1], w[k][2]);
        const float c01 = volume_lerp(c[k][2], c[k][3], w[k][2]);
        const float c10 = volume_lerp(c[k][4], c[k][5], w[k][2]);
        const float c11 = volume_lerp(c[k][6], c[k][7], w[k][2]);
        out[k] = volume_lerp(volume_lerp(c00, c01, w[k][1]), volume_lerp(c10, c11, w[k][1]), w[k][0]);
    }
}

// Both trackers advance by distances that depend on the random numbers alone,
// so a lane that waits for its voxels can have the next steps' in flight too:
// with AHEAD > 1 (counter-based draws, which can be given back) they read AHEAD
// steps at once and then take them in order, giving back the draws of steps not
// taken. Distances and draws are those of one step at a time.
template <class Rng>
MC_D float volume_step(float t, float majorant, Rng& rng) {
    return t - logf(1.0f - rng.uniform()) / majorant;
}

// PT:796-815 delta tracking: the distance of the first real collision along
// o + d t, or maxDistance when the ray leaves the medium without one.
template <int AHEAD, class Rng>
MC_D float volume_free_flight(const mc_volume_grid* g, float extinctionScale, float gridMax, const V3& o, const V3& d,
                              float maxDistance, Rng& rng) {
    const float majorant = extinctionScale * gridMax;
    if (!(majorant > 0.0f)) return maxDistance;
    float t = 0.0f;
    if constexpr (AHEAD > 1) {
        for (int step = 0; step < 8192; step += AHEAD) {
            float at[AHEAD], u[AHEAD], density[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; k++) {
                t = at[k] = volume_step(t, majorant, rng);
                u[k] = rng.uniform();
            }
            volume_densities<AHEAD>(g, o, d, at, maxDistance, density);
#pragma unroll
            for (int k = 0; k < AHEAD; k++) {
                if (at[k] >= maxDistance) {
                    rng.give_back(2 * (AHEAD - k) - 1);
                    return maxDistance;
                }
                if (u[k] < density[k] / gridMax) {
                    rng.give_back(2 * (AHEAD - k) - 2);
                    return at[k];
                }
            }
        }
        return maxDistance;
    }
    for (int step = 0; step < 8192; step++) {
        t = volume_step(t, majorant, rng);
        if (t >= maxDistance) return maxDistance;
        const float density = volume_density(g, o + d * t);
        if (rng.uniform() < density / gridMax) return t;
    }
    return maxDistance;
}

// PT:817-838 ratio tracking: the transmittance of the segment o + d t, t in
// [0, length), as the product of (1 - density / majorant) at the tentative
// collisions; 0 once it falls below 1e-4.
template <int AHEAD, class Rng>
MC_D float volume_transmittance(const mc_volume_grid* g, float extinctionScale, float gridMax, const V3& o, const V3& d,
                                float length, Rng& rng) {
    const float majorant = extinctionScale * gridMax;
    if (!(majorant > 0.0f)) return 1.0f;
    float T = 1.0f;
    float t = 0.0f;
    if constexpr (AHEAD > 1) {
        for (int step = 0; step < 8192; step += AHEAD) {
            float at[AHEAD], density[AHEAD];
#pragma unroll
            for (int k = 0; k < AHEAD; k++) t = at[k] = volume_step(t, majorant, rng);
            volume_densities<AHEAD>(g, o, d, at, length, density);
#pragma unroll
            for (int k = 0; k < AHEAD; k++) {
                if (at[k] >= length) {
                    rng.give_back(AHEAD - 1 - k);
                    return T;
                }
                T = T * (1.0f - density[k] / gridMax);
                if (T < 1e-4f) {
                    rng.give_back(AHEAD - 1 - k);
                    return 0.0f;
                }
            }
        }
        return T;
    }
    for (int step = 0; step < 8192; step++) {
        t = volume_step(t, majorant, rng);
        if (t >= length) break;
        const float density = volume_density(g, o + d * t);
        T = T * (1.0f - density / gridMax);
        if (T < 1e-4f) return 0.0f;
    }
    return T;
}

}  // namespace mc
