// Photon state and the steps of the walk shared by the transport kernel (one photon per thread) and the
// tail kernel (one photon per group of 8 lanes): voxel index, detector search and tallies, plane crossings, launch,
// boundary crossing and the biased spin. Both kernels inline the same arithmetic, so a photon takes the
// same path in either.
#pragma once

#include <cstdint>
#include <type_traits>

#include "geom.cuh"
#include "photon.cuh"
#include "xmc_internal.h"

namespace xmc {

namespace {

constexpr unsigned FULL = 0xffffffffu;

// Photon weight in 2^31 fixed point: 32 bits (weight <= 1 always holds without biasing) or 64 bits
// (the biasing factor W / p can raise a weight above 1).
template <typename WT>
struct Photon {
    float px, py, pz, dx, dy, dz;
    float time, trange, orange;
    WT w;
    int layer;
    uint32_t visited;
    uint32_t iter;
    int excl;
    float tmin;
    float gap_lo, gap_hi;  // triangle-free z-gap containing the photon (empty if none)
    int rdet;              // replay pass: the detector this photon reached in the run pass
    unsigned long long pid;
};

__device__ __forceinline__ float w2f(uint32_t w) { return __uint2float_rn(w); }
__device__ __forceinline__ float w2f(unsigned long long w) { return __ull2float_rn(w); }
template <typename WT> __device__ __forceinline__ WT f2w(float f);
template <> __device__ __forceinline__ uint32_t f2w<uint32_t>(float f) { return __float2uint_rn(f); }
template <> __device__ __forceinline__ unsigned long long f2w<unsigned long long>(float f) { return __float2ull_rn(f); }
// w^2 in fixed point ((w w) >> 31), exact for weights below 2^32 in weight units
__device__ __forceinline__ unsigned long long wsq(uint32_t w) { return ((unsigned long long)w * w) >> 31; }
__device__ __forceinline__ unsigned long long wsq(unsigned long long w) { return (__umul64hi(w, w) << 33) | ((w * w) >> 31); }

// The triangle-free z-gap around z: (highest occupied top below z, lowest occupied bottom above
// z), or an empty interval when z lies inside an occupied slab.
__device__ __forceinline__ void find_gap(const float* __restrict__ zlo, const float* __restrict__ zhi, int n, float z,
                                         float& glo, float& ghi) {
    glo = -INFINITY;
    ghi = INFINITY;
    for (int i = 0; i < n; ++i) {
        if (z >= zlo[i] && z <= zhi[i]) {
            glo = INFINITY;
            ghi = -INFINITY;
            return;
        }
        if (zhi[i] < z) glo = fmaxf(glo, zhi[i]);
        if (zlo[i] > z) ghi = fminf(ghi, zlo[i]);
    }
}

// GetAreaIndex (mcml_kernel.cpp:190-227): voxel of a point, -1 outside Area. `tol` (voxel units)
// widens the box for points on a surface: the reference stops 1e-10 mm in front of a surface
// (mcml_kernel.cpp:60,87), so a surface lying on an Area face counts as inside; the FP32 hit point
// sits on the surface within rounding and is accepted within tol, clamped to the edge voxel.
__device__ __forceinline__ int area_index(const KParams& P, float x, float y, float z, float tol) {
    float fx = (x - P.ax) * P.asx, fy = (y - P.ay) * P.asy, fz = (z - P.az) * P.asz;
    if (!(fx >= -tol && fy >= -tol && fz >= -tol)) return -1;
    if (!(fx < (float)P.nx + tol && fy < (float)P.ny + tol && fz < (float)P.nz + tol)) return -1;
    const int ix = min(max((int)fx, 0), P.nx - 1), iy = min(max((int)fy, 0), P.ny - 1), iz = min(max((int)fz, 0), P.nz - 1);
    if (P.byte_sentinel && ix == 255 && iy == 255 && iz == 255) return -1;
    return (ix * P.ny + iy) * P.nz + iz;
}

// Block-private tallies in shared memory.
struct SmemTally {
    unsigned long long* ledger;  // [kLedgerSlots]
    unsigned long long* det;     // [n_dets * 4]
};

__device__ __forceinline__ void lat(unsigned long long* p, unsigned long long v) {
    if (v) atomicAdd(p, v);
}

// mcml_kernel.cpp:663-742 (first matching cube, then ring; layer filter; angle test) and the
// detector tallies of :744-858. Weight arithmetic in fixed point.
template <class Ph>
__device__ int find_detector(const KParams& P, const DevDetector* __restrict__ s_det, const Ph& ph) {
    int det = -1;
    const float l2 = __fmaf_rn(ph.dz, ph.dz, __fmaf_rn(ph.dx, ph.dx, __fmul_rn(ph.dy, ph.dy)));
    const float ac = -ph.dz / l2;
    const int n_scan = P.rings_sorted ? P.n_cubes : P.n_dets;
    for (int i = 0; i < n_scan; ++i) {
        const DevDetector D = s_det[i];
        bool inside;
        if (i < P.n_cubes) {
            inside = ph.px >= D.cx - D.hx && ph.px < D.cx + D.hx && ph.py >= D.cy - D.hy && ph.py < D.cy + D.hy &&
                     ph.pz >= D.cz - D.hz && ph.pz < D.cz + D.hz;
        } else {
            const float ex = ph.px - D.cx, ey = ph.py - D.cy;
            const float r = radius_xy(ex, ey);
            inside = r >= D.hx && r < D.hy;
        }
        if (inside && (D.filter & ph.visited) && ac > D.cos_angle) {
            det = i;
            break;
        }
    }
    if (det < 0 && P.rings_sorted) {
        // concentric, sorted, non-overlapping rings: the only ring that can contain the radius is
        // the last one whose small radius is <= r, so the first match of the scan is this one
        const DevDetector* R = s_det + P.n_cubes;
        const float ex = ph.px - R[0].cx, ey = ph.py - R[0].cy;
        const float r = radius_xy(ex, ey);
        int lo = 0, hi = P.n_rings - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (R[mid].hx <= r) lo = mid;
            else hi = mid - 1;
        }
        const DevDetector D = R[lo];
        if (r >= D.hx && r < D.hy && (D.filter & ph.visited) && ac > D.cos_angle) det = P.n_cubes + lo;
    }
    return det;
}

template <class Ph>
__device__ void tally_detection(const KParams& P, const SmemTally& S, const Ph& ph, int det) {
    using WT = decltype(ph.w);
    const WT w = ph.w;
    const float total = ph.trange + ph.orange;
    const WT tw = total > 0.0f ? f2w<WT>(w2f(w) * (ph.trange / total)) : (WT)0;
    const unsigned long long w2 = wsq(w);
    atomicAdd(&S.det[4 * det + 0], (unsigned long long)w);
    atomicAdd(&S.det[4 * det + 1], 1ull);
    lat(&S.det[4 * det + 2], tw);
    lat(&S.det[4 * det + 3], w2);
    atomicAdd(&S.ledger[L_N_DETECTED], 1ull);
    // time bins (mcml_kernel.cpp:812-849): [t0 + i dt, t0 + (i+1) dt), last bin open-ended
    if (ph.time >= P.t0) {
        int bin = P.n_time - 1;
        if (P.dt > 0.0f) {
            const float f = (ph.time - P.t0) / P.dt;
            if (f < (float)(P.n_time - 1)) bin = (int)f;
        }
        unsigned long long* tb = P.tbin + 4 * ((size_t)det * P.n_time + bin);
        atomicAdd(tb + 0, (unsigned long long)w);
        atomicAdd(tb + 1, 1ull);
        lat(tb + 2, tw);
        lat(tb + 3, w2);
    }
}

// A detected photon whose crossing log overflowed: walked again by the replay pass.
__device__ __forceinline__ void list_for_replay(const KParams& P, unsigned long long pid, int det) {
    const unsigned long long slot = atomicAdd(P.replay_count, 1ull);
    if (slot < P.replay_cap) P.replay_list[slot] = ((pid - P.first_id) << 16) | (unsigned long long)det;
}

// UpdatePhotonTrajectory (mcml_kernel.cpp:750-792): for a move from p0 to p1, every z-plane through
// voxel centres between them (inside Area) is crossed at one voxel. The run pass adds the photon's
// weight to the scattering map there and appends the voxel to the thread's crossing log (`xl`, `xn`
// entries so far, counted past the capacity so that an overflow shows); at detection the log is
// counted in the detector's trajectory map (UpdateDetectorTrajectory, :794-810, which walks the
// reference's per-photon PhotonTrajectory the same way). The replay pass, for photons whose log
// overflowed, counts each crossing in the map of the detector the photon reached.
// Row of the crossing log of thread `thread` of this block.
__device__ __forceinline__ unsigned* xlog_row(const KParams& P, unsigned thread) {
    return P.xlog + ((size_t)blockIdx.x * blockDim.x + thread) * P.xlog_cap;
}

__device__ void cross_planes(const KParams& P, float x0, float y0, float z0, float x1, float y1, float z1,
                             unsigned long long w, int rdet, unsigned* __restrict__ xl, unsigned& xn,
                             unsigned& n_cross) {
    if (z1 == z0) return;
    // first plane at or above the lower end of the move; most moves cross none and stop here
    const float step = P.plane_dz;
    const int k = (int)fmaf(fminf(z0, z1) - P.az, P.asz, 0.5f);
    float plane = P.az + k * step + 0.5f * step;
    if (plane > fmaxf(z0, z1) || plane >= P.area_zend) return;
    float sx = x0, sy = y0, sz = z0, fz = z1, ex = x1 - x0, ey = y1 - y0, ez = z1 - z0;
    if (z1 < z0) {
        sx = x1; sy = y1; sz = z1; fz = z0;
        ex = -ex; ey = -ey; ez = -ez;
    }
    const float inv = 1.0f / ez;
    for (int guard = 0; plane <= fz && plane < P.area_zend && guard < 65536; ++guard) {
        const float t = (plane - sz) * inv;
        const int idx = area_index(P, fmaf(ex, t, sx), fmaf(ey, t, sy), plane, 0.0f);
        if (idx < 0) break;
        ++n_cross;
        if (P.mode == 0) {
            if (w && P.scatter) atomicAdd(&P.scatter[idx], (unsigned long long)w);
            if (xl) {
                if (xn < P.xlog_cap) xl[xn] = (unsigned)idx;
                xn += xn <= P.xlog_cap;  // saturates at capacity + 1: overflowed
            }
        } else {
            atomicAdd(&P.traj[(size_t)rdet * P.grid + idx], 1ull);
        }
        plane += step;
    }
}

__device__ __forceinline__ unsigned long long pack_hit(float d, unsigned tri) {
    return ((unsigned long long)__float_as_uint(d) << 32) | tri;
}

template <class Ph>
__device__ __forceinline__ void kill(const SmemTally& S, Ph& ph, bool& alive, int count_slot, int weight_slot) {
    atomicAdd(&S.ledger[count_slot], 1ull);
    lat(&S.ledger[weight_slot], ph.w);
    atomicAdd(&S.ledger[L_TERMINATED], 1ull);
    alive = false;
}

template <class Ph>
__device__ __forceinline__ void launch_photon(const KParams& P, Ph& ph, unsigned long long pid) {
    ph.pid = pid;
    ph.px = P.sx;
    ph.py = P.sy;
    ph.pz = P.sz;
    if (P.beam_radius > 0.0f) {
        const uint4 r = philox4x32_10(make_uint4((uint32_t)pid, (uint32_t)(pid >> 32), 0u, 1u), P.keys);
        const float rad = P.beam_radius * sqrtf(u24(r.x));
        float a = u24(r.y);
        a = a > 0.5f ? a - 1.0f : a;
        float sp, cp;
        __sincosf(6.283185307179586f * a, &sp, &cp);
        ph.px += rad * cp;
        ph.py += rad * sp;
    }
    ph.dx = P.dx;
    ph.dy = P.dy;
    ph.dz = P.dz;
    ph.time = 0.0f;
    ph.trange = 0.0f;
    ph.orange = 0.0f;
    ph.w = P.w0;
    ph.layer = 1;
    ph.visited = 1u << 1;
    ph.iter = 0;
    ph.excl = -1;
    ph.tmin = kTminAfter;
}

constexpr uint32_t kBiasMaxTrials = 65536;

// ComputePhotonDirectionWithBiasing (mcml_kernel.cpp:398-428): the local attractive direction v
// (GetLocalAttractiveVector, :325-364: normalised difference of the fields of two point sources on
// the vertical through the target point, l_tr above it and l_tr + 2 delta below it), a new direction
// by rejection from HG with acceptance p = (0.1 + 0.45 (1 + d.v))^attractiveFactor (trial k draws the
// Philox block (id, iteration, 2 + k): slot 0 cos theta, slot 1 azimuth, slot 2 acceptance), and
// the weight factor W(d_old.v) / p from the layer's weight-integral table (nearest node).
// kLanes > 1: a group of that many lanes holds this photon and draws that many trials at once; the first
// accepted one counts.
template <int kLanes, class Ph>
__device__ __forceinline__ void biased_spin(const KParams& P, const DevLayer& L, int layer, Ph& ph,
                                            unsigned long long& gained, unsigned long long& lost) {
    using WT = decltype(ph.w);
    const float ltr = 3.0f * (1.0f / (3.0f * ((1.0f - L.g) * L.mus + L.mua)));
    const float delta = 0.74f * ltr;
    const float rx = ph.px - P.bias_ox, ry = ph.py - P.bias_oy, rz = ph.pz - P.bias_oz;
    const float ex = rx - P.bias_rx, ey = ry - P.bias_ry;
    const float az = rz - (P.bias_rz + ltr), bz = rz - (P.bias_rz - ltr - 2.0f * delta);
    const float ia = rsqrtf(dot3(ex, ey, az, ex, ey, az)), ib = rsqrtf(dot3(ex, ey, bz, ex, ey, bz));
    const float ca = ia * ia * ia, cb = ib * ib * ib;
    float vx = ex * (cb - ca), vy = ey * (cb - ca), vz = diff2(bz, cb, az, ca);
    const float vn = rsqrtf(dot3(vx, vy, vz, vx, vy, vz));
    vx *= vn; vy *= vn; vz *= vn;
    const int t = P.layer_wtab[layer];
    auto integral = [&]() {
        const float step = 2.0f / (float)(P.wtab_n - 1);
        int e = (int)floorf((dot3(ph.dx, ph.dy, ph.dz, vx, vy, vz) + 1.0f) / step + 0.5f);
        e = min(max(e, 0), P.wtab_n - 1);
        return __ldg(&P.wtab[(size_t)t * P.wtab_n + e]);
    };
    float W = 0.0f;
    // on its way while the trials are drawn (tail kernel, 50,000 photons: 2.87 -> 2.81 ms); in the transport kernel, which
    // is short of registers, after them (5e5 photons: 10.9 ms, 11.1 the other way)
    if constexpr (kLanes > 1)
        if (t >= 0) W = integral();
    float nx = ph.dx, ny = ph.dy, nz = ph.dz, p = 1.0f;
    for (uint32_t k = threadIdx.x & (kLanes - 1); k < kBiasMaxTrials; k += kLanes) {
        const uint4 r = philox4x32_10(make_uint4((uint32_t)ph.pid, (uint32_t)(ph.pid >> 32), ph.iter - 1u, 2u + k),
                                      P.keys);
        nx = ph.dx; ny = ph.dy; nz = ph.dz;
        hg_spin(L.hg_a, L.hg_b, L.hg_c, L.hg_d, L.hg_e, u24(r.x), u24(r.y), nx, ny, nz);
        p = powf(fmaf(0.45f, 1.0f + dot3(nx, ny, nz, vx, vy, vz), 0.1f), P.bias_eps);
        if constexpr (kLanes > 1) {
            const unsigned first = threadIdx.x & 31u & ~(kLanes - 1u);
            const unsigned group = (unsigned)((1ull << kLanes) - 1ull) << first;
            const unsigned acc = __ballot_sync(group, p > u24(r.z)) >> first;
            if (acc == 0u && k / kLanes + 1u < kBiasMaxTrials / kLanes) continue;
            const int src = acc ? __ffs(acc) - 1 : kLanes - 1;  // none of all trials: the last one stands
            nx = __shfl_sync(group, nx, src, kLanes);
            ny = __shfl_sync(group, ny, src, kLanes);
            nz = __shfl_sync(group, nz, src, kLanes);
            p = __shfl_sync(group, p, src, kLanes);
            break;
        }
        if (p > u24(r.z)) break;
    }
    if (t >= 0) {
        if constexpr (kLanes == 1) W = integral();
        const WT nw = f2w<WT>(w2f(ph.w) * (W / p));
        if (nw > ph.w) gained += nw - ph.w;
        else lost += ph.w - nw;
        ph.w = nw;
    }
    ph.dx = nx; ph.dy = ny; ph.dz = nz;
}

// Whether a step that passes over the z-range [pz, zend] stays in the photon's triangle-free z-gap.
template <class Ph>
__device__ __forceinline__ bool in_gap(const Ph& ph, float zend) {
    return (fminf(ph.pz, zend) > ph.gap_lo) & (fmaxf(ph.pz, zend) < ph.gap_hi);
}

// An interaction step that needs no ray query (it stays inside the photon's triangle-free z-gap, or clear of
// every triangle), does not end outside Area where that kills, and leaves the weight at or above the cut: moves the photon and drops `dw`
// into voxel `idx` (-1: outside Area). False, with nothing changed, for any other step.
template <class Ph, typename WT>
__device__ __forceinline__ bool free_step(const KParams& P, const DevLayer& L, float step, bool area_kill, Ph& ph, int& idx,
                                          WT& dw) {
    const float zend = fmaf(step + kStepExtend, ph.dz, ph.pz);
    const float nx = fmaf(step, ph.dx, ph.px), ny = fmaf(step, ph.dy, ph.py), nz = fmaf(step, ph.dz, ph.pz);
    // area_index with tol 0 and no branch: inside Area the coordinates are in [0, 4096), so that adding 2^23
    // towards zero leaves their integer parts in the float's low bits, and the bits above cancel in voxel_bias
    const float fx = (nx - P.ax) * P.asx, fy = (ny - P.ay) * P.asy, fz = (nz - P.az) * P.asz;
    const bool inside = (fx >= 0.0f) & (fy >= 0.0f) & (fz >= 0.0f) & (fx < (float)P.nx) & (fy < (float)P.ny) & (fz < (float)P.nz);
    const uint32_t bx = __float_as_uint(__fadd_rz(fx, 8388608.0f)), by = __float_as_uint(__fadd_rz(fy, 8388608.0f));
    const uint32_t voxel = (bx * (uint32_t)P.ny + by) * (uint32_t)P.nz + __float_as_uint(__fadd_rz(fz, 8388608.0f)) + P.voxel_bias;
    idx = inside & (voxel != P.voxel_sentinel) ? (int)voxel : -1;
    dw = f2w<WT>(w2f(ph.w) * L.absorb);
    dw = min(dw, ph.w);
    if ((idx < 0) & area_kill | (ph.w - dw < P.w_min) | (ph.iter >= P.max_steps) | (L.glass != 0)) return false;
    if (!in_gap(ph, zend) && !clear_segment(P, ph.px, ph.py, ph.pz, fmaf(step + kStepExtend, ph.dx, ph.px),
                                            fmaf(step + kStepExtend, ph.dy, ph.py), zend))
        return false;
    ph.px = nx;
    ph.py = ny;
    ph.pz = nz;
    ph.time = fmaf(step, L.n, ph.time);
    if ((P.target_mask >> ph.layer) & 1u) ph.trange += step;
    else ph.orange += step;
    ph.w -= dw;
    ph.excl = -1;
    ph.tmin = 0.0f;
    ph.iter++;
    return true;
}

// CrossBoundary (mcml_kernel.cpp:229-284) at triangle `tri`, hit from layer L: Fresnel test against
// `u_fresnel`, then refraction or reflection. Returns kCrossInvalid when the surface leads nowhere from
// this layer, kCrossLeft when the photon leaves the tissue (its direction unchanged, for the detectors),
// else kCrossInside with the photon's direction and layer updated.
enum { kCrossInvalid = -1, kCrossLeft = 0, kCrossInside = 1 };

template <class Ph>
__device__ __forceinline__ int cross_boundary(const KParams& P, const DevLayer* s_layer, const float4* s_tris,
                                              const int8_t* s_next, const DevLayer& L, int tri, float u_fresnel, Ph& ph) {
    const float4 a = tri < P.smem_tris ? s_tris[3 * tri] : __ldg(&P.tris[3 * tri]);
    const float4 b = tri < P.smem_tris ? s_tris[3 * tri + 1] : __ldg(&P.tris[3 * tri + 1]);
    const float4 c = tri < P.smem_tris ? s_tris[3 * tri + 2] : __ldg(&P.tris[3 * tri + 2]);
    // GetPlaneNormal (mcml_math.cpp:45-50), normalised
    const float e1x = a.x - b.x, e1y = a.y - b.y, e1z = a.z - b.z;
    const float e2x = a.x - c.x, e2y = a.y - c.y, e2z = a.z - c.z;
    float nx = diff2(e1y, e2z, e1z, e2y), ny = diff2(e1z, e2x, e1x, e2z), nz = diff2(e1x, e2y, e1y, e2x);
    const float nr = rsqrtf(dot3(nx, ny, nz, nx, ny, nz));
    nx *= nr; ny *= nr; nz *= nr;
    const int surf = __float_as_int(a.w);
    const int next = surf * MAX_LAYERS + ph.layer < P.smem_next ? (int)s_next[surf * MAX_LAYERS + ph.layer]
                                                                 : (int)__ldg(&P.next_layer[surf * MAX_LAYERS + ph.layer]);
    if (next < 0) return kCrossInvalid;
    const float ni = L.n, nt = s_layer[next].n;
    const float dn = dot3(ph.dx, ph.dy, ph.dz, nx, ny, nz);
    const float R = fresnel_reflectance(ni, nt, fabsf(dn));
    if (u_fresnel > R) {
        if (next == 0) return kCrossLeft;
        // RefractVector (mcml_kernel.cpp:595-616)
        const float six = mul_rn(ni, ph.dx), siy = mul_rn(ni, ph.dy), siz = mul_rn(ni, ph.dz);
        const float t1 = dot3(six, siy, siz, nx, ny, nz);
        float t2 = sqrtf(diff2(nt, nt, ni, ni) / (t1 * t1) + 1.0f);
        t2 = (t2 - 1.0f) * t1;
        float ox = fmaf(t2, nx, six), oy = fmaf(t2, ny, siy), oz = fmaf(t2, nz, siz);
        const float on = rsqrtf(dot3(ox, oy, oz, ox, oy, oz));
        ph.dx = ox * on; ph.dy = oy * on; ph.dz = oz * on;
        ph.layer = next;
        ph.visited |= 1u << next;
    } else {
        // ReflectVector (mcml_kernel.cpp:582-593)
        const float t = 2.0f * dn;
        float ox = fmaf(-t, nx, ph.dx), oy = fmaf(-t, ny, ph.dy), oz = fmaf(-t, nz, ph.dz);
        const float on = rsqrtf(dot3(ox, oy, oz, ox, oy, oz));
        ph.dx = ox * on; ph.dy = oy * on; ph.dz = oz * on;
    }
    ph.excl = tri;
    ph.tmin = kTminAfter;
    return kCrossInside;
}

}  // namespace

}  // namespace xmc
