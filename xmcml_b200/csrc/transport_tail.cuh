// Tail kernel of a transport run: one photon per group of kTailGroup lanes.
//
// Once the photon ids are used up, the transport kernel's warps run on with the few lanes whose walks are
// long, and a step of such a warp takes thousands of cycles with one live lane as with 32 (10 dependent
// Philox rounds, the logarithm, the angles and the optics one after the other); a run that has few photons
// to begin with is all tail. Those photons come here (TailPhoton list, or the id dispenser itself for runs
// that are given to this kernel whole, xmc_internal.h whole_in_tail_max) and a group of lanes walks each of them:
//   * the random numbers do not depend on the path, so the lanes draw 16 iterations at once, each lane the
//     Philox blocks of two of them with their logarithms, Henyey-Greenstein angles and azimuths;
//   * a step that needs no ray query (free_step) is a short chain that every lane of the group runs on the
//     same values and that a single branch leaves;
//   * a ray query tests one candidate triangle per lane, and a biased spin draws 8 trials at once.
// The arithmetic is the transport kernel's (walk.cuh, photon.cuh), so every tally is the same bit for bit.
//
// What bounds it: the latency of one step, 0.4 us of a lone photon (1.5 us in a warp of the transport kernel).
// Groups of 8 lanes beat whole warps (more photons for the same chain; planar stack with roulette, 1e6
// photons 47.5 -> 43.8 ms when this was the only change) and groups of 4 or 16; 2 blocks per SM at 128
// registers beat 3 at 80 (spills). A warp hands its photons over when at most 8 lanes hold one: 4 and 16
// were within 3 % and slower. Handing over every photon of 1,500 or 4,000 steps at once made it slower (29.8
// and 31.5 ms against 28.6): here most photons are long walks. B200: 2e4 photons into the planar stack
// 5.6 -> 1.75 ms, 901 under a glass cover 4.2 -> 0.9 ms; of runs of 1e6 photons it takes most of the part that does
// not grow with their number: 6.5 ms of the planar stack's 27, 7.8 of the height field's 39, 9.0 of the ellipsoid's 48,
// 2.1 of the glass cover's 13.
#pragma once

#include "walk.cuh"

namespace xmc {

namespace {

constexpr int kTailThreads = 256;
constexpr int kTailWarps = kTailThreads / 32;
constexpr int kTailGroup = 8;  // lanes per photon (a power of two)

constexpr int kTailDraws = 2;  // iterations that each lane draws at a time

// The draws of a warp's groups: {step length, cos theta, sin theta, sin azimuth}, cos azimuth.
struct TailDraws {
    float4 a[32 * kTailDraws];
    float cp[32 * kTailDraws];
};

struct TailLayout {
    size_t nodes, tris, layer, det, next, draws, bytes;
};
__host__ __device__ inline TailLayout tail_layout(const KParams& P) {
    TailLayout l;
    l.nodes = sizeof(unsigned long long) * (size_t)(kLedgerSlots + 4 * P.n_dets);
    l.tris = l.nodes + sizeof(float4) * 2 * (size_t)P.smem_nodes;
    l.layer = l.tris + sizeof(float4) * 3 * (size_t)P.smem_tris;
    l.det = l.layer + sizeof(DevLayer) * MAX_LAYERS;
    l.next = l.det + sizeof(DevDetector) * (size_t)P.n_dets;
    l.draws = (l.next + (size_t)P.smem_next + 15) & ~(size_t)15;
    l.bytes = l.draws + sizeof(TailDraws) * kTailWarps;
    return l;
}

// The lanes of the calling thread's group.
__device__ __forceinline__ unsigned tail_group_mask() {
    return (unsigned)((1ull << kTailGroup) - 1ull) << (threadIdx.x & 31 & ~(kTailGroup - 1));
}

// Nearest hit with tmin <= t <= tmax of one ray that all lanes of a group hold, over the big triangles and the entries
// of the cells under the segment, one candidate per lane: the candidates and the choice of grid_nearest
// (geom.cuh). False when the segment covers more cells than the group has lanes (the caller uses the BVH).
__device__ __forceinline__ bool tail_grid_query(const KParams& P, const float4* __restrict__ s_big,
                                                const float4* __restrict__ s_tris, float ox, float oy, float oz, float dx,
                                                float dy, float dz, float tmin, float tmax, int excl, Hit& hit,
                                                unsigned& retests, unsigned& n_visit, unsigned& n_tri) {
    constexpr int G = kTailGroup;
    const int lane = threadIdx.x & (G - 1);
    const unsigned gm = tail_group_mask();
    const float ex = fmaf(dx, tmax, ox), ey = fmaf(dy, tmax, oy), ez = fmaf(dz, tmax, oz);
    const float fx0 = fminf(fmaxf((fminf(ox, ex) - P.grid_x0) * P.grid_icx, -1.0f), (float)P.grid_nx);
    const float fx1 = fminf(fmaxf((fmaxf(ox, ex) - P.grid_x0) * P.grid_icx, -1.0f), (float)P.grid_nx);
    const float fy0 = fminf(fmaxf((fminf(oy, ey) - P.grid_y0) * P.grid_icy, -1.0f), (float)P.grid_ny);
    const float fy1 = fminf(fmaxf((fmaxf(oy, ey) - P.grid_y0) * P.grid_icy, -1.0f), (float)P.grid_ny);
    const bool inside = fx1 >= 0.0f && fy1 >= 0.0f && fx0 < (float)P.grid_nx && fy0 < (float)P.grid_ny;
    const int i0 = max(0, (int)floorf(fx0)), i1 = min(P.grid_nx - 1, (int)floorf(fx1));
    const int j0 = max(0, (int)floorf(fy0)), j1 = min(P.grid_ny - 1, (int)floorf(fy1));
    const int ww = i1 - i0 + 1, ncell = inside ? ww * (j1 - j0 + 1) : 0;
    if (ncell > G) return false;
    const float zl = fminf(oz, ez), zh = fmaxf(oz, ez);
    // this lane's cell: its entries that the segment's z-range can meet (cells_runs: per z-interval)
    uint2 cell = make_uint2(0u, 0u);
    if (lane < ncell) {
        const unsigned ci = (unsigned)(j0 + lane / ww) * (unsigned)P.grid_nx + (unsigned)(i0 + lane % ww);
        cell = __ldg(&P.cells[ci]);
        const float4 za = __ldg(&P.cell_z[2 * ci]), zb = __ldg(&P.cell_z[2 * ci + 1]);
        if ((za.y < zl || za.x > zh) && (za.w < zl || za.z > zh) && (zb.y < zl || zb.x > zh) && (zb.w < zl || zb.z > zh))
            cell.y = 0u;
        ++n_visit;
    }
    unsigned best_d = __float_as_uint(tmax), best_t = 0xffffffffu;
    auto candidate = [&](float4 a, float4 b, float4 c, int t) {
        ++n_tri;
        const float d = __fadd_rn(tri_distance(a, b, c, ox, oy, oz, dx, dy, dz, retests), 0.0f);
        if (d >= tmin && d <= tmax && pack_hit(d, (unsigned)t) < (((unsigned long long)best_d << 32) | best_t)) {
            best_d = __float_as_uint(d);
            best_t = (unsigned)t;
        }
    };
    for (int k = lane; k < P.n_big; k += G) {
        const float4 en = s_big[4 * k];
        const int t = f2i(en.z);
        if (en.y < zl || en.x > zh || t == excl) continue;
        candidate(s_big[4 * k + 1], s_big[4 * k + 2], s_big[4 * k + 3], t);
    }
    for (int c = 0; c < ncell; ++c) {
        const unsigned at = __shfl_sync(gm, cell.x, c, G), end = at + __shfl_sync(gm, cell.y, c, G);
        for (unsigned k = at + lane; k < end; k += G) {
            const float4 en = __ldg(&P.cell_entries[k]);
            const int t = f2i(en.z);
            if (en.y < zl || en.x > zh || t == excl) continue;
            if (t < P.smem_tris) candidate(s_tris[3 * t], s_tris[3 * t + 1], s_tris[3 * t + 2], t);
            else candidate(__ldg(&P.tris[3 * t]), __ldg(&P.tris[3 * t + 1]), __ldg(&P.tris[3 * t + 2]), t);
        }
    }
    __syncwarp(gm);
    const unsigned d = __reduce_min_sync(gm, best_d);
    const unsigned t = __reduce_min_sync(gm, best_d == d ? best_t : 0xffffffffu);
    hit.tri = (int)t;  // -1: none
    hit.t = __uint_as_float(d);
    return true;
}

}  // namespace

template <bool kBias, bool kLog>
__global__ void __launch_bounds__(kTailThreads, 2) transport_tail_kernel(const KParams P) {
    using WT = typename std::conditional<kBias, unsigned long long, uint32_t>::type;
    const unsigned n_listed = P.tail_direct ? 0u : *P.tail_count;
    constexpr int G = kTailGroup, D = G * kTailDraws;
    if (!P.tail_direct && blockIdx.x >= n_listed) return;  // nothing for this block
    extern __shared__ __align__(16) unsigned char smem[];
    const TailLayout lay = tail_layout(P);
    unsigned long long* s_ledger = reinterpret_cast<unsigned long long*>(smem);
    unsigned long long* s_dettal = s_ledger + kLedgerSlots;
    float4* s_nodes = reinterpret_cast<float4*>(smem + lay.nodes);
    float4* s_tris = reinterpret_cast<float4*>(smem + lay.tris);
    DevLayer* s_layer = reinterpret_cast<DevLayer*>(smem + lay.layer);
    DevDetector* s_det = reinterpret_cast<DevDetector*>(smem + lay.det);
    int8_t* s_next = reinterpret_cast<int8_t*>(smem + lay.next);
    TailDraws& W = reinterpret_cast<TailDraws*>(smem + lay.draws)[threadIdx.x >> 5];
    float4* const draw = W.a + (threadIdx.x & 31) / G * D;
    float* const draw_cp = W.cp + (threadIdx.x & 31) / G * D;
    __shared__ float s_zlo[kMaxZSlabs], s_zhi[kMaxZSlabs];
    __shared__ float4 s_big[4 * kMaxBigTriangles];
    for (int i = threadIdx.x; i < 4 * P.n_big; i += blockDim.x) s_big[i] = P.big[i];
    for (int i = threadIdx.x; i < P.n_zocc; i += blockDim.x) {
        s_zlo[i] = P.zocc_lo[i];
        s_zhi[i] = P.zocc_hi[i];
    }
    for (int i = threadIdx.x; i < kLedgerSlots + 4 * P.n_dets; i += blockDim.x) s_ledger[i] = 0ull;
    for (int i = threadIdx.x; i < 2 * P.smem_nodes; i += blockDim.x) s_nodes[i] = __ldg(&P.nodes[i]);
    for (int i = threadIdx.x; i < 3 * P.smem_tris; i += blockDim.x) s_tris[i] = __ldg(&P.tris[i]);
    for (int i = threadIdx.x; i < MAX_LAYERS; i += blockDim.x) s_layer[i] = P.layer[i];
    for (int i = threadIdx.x; i < P.n_dets; i += blockDim.x) s_det[i] = P.dets[i];
    for (int i = threadIdx.x; i < P.smem_next; i += blockDim.x) s_next[i] = P.next_layer[i];
    __syncthreads();
    const SmemTally S{s_ledger, s_dettal};

    const int lane = threadIdx.x & (G - 1), first = threadIdx.x & 31 & ~(G - 1);  // of the group; its first lane
    const unsigned gm = tail_group_mask();
    const bool lead = lane == 0;  // the lane that adds the photon's tallies
    const bool area_kill = !(P.flags & XMC_NO_AREA_KILL);
    const bool roulette = (P.flags & XMC_ROULETTE) != 0;
    const bool record_planes = P.mode == 1 || (P.flags & XMC_SCATTERING_MAP) != 0 || kLog;
    unsigned retests = 0, n_visit = 0, n_tri = 0, n_cross = 0;
    unsigned long long bias_gained = 0, bias_lost = 0;
    unsigned long long absorbed = 0, absorbed_out = 0, absorbed_tgt = 0;
    unsigned budget_hit = 0;

    // the first photons are dealt over the blocks, then over a block's warps, then over a warp's groups, so that
    // few photons run on as many schedulers as there are; the rest come from the dispensers
    const unsigned warps = gridDim.x * kTailWarps, n_groups = warps * (32 / G);
    unsigned long long next = (unsigned long long)(first / G) * warps + (threadIdx.x / 32) * gridDim.x + blockIdx.x;
    const unsigned long long n_next = P.tail_direct ? P.n_photons : (unsigned long long)n_listed;
    bool dealt = true, done = false;

    Photon<WT> ph;
    unsigned xrow = 0, xn = 0;
    bool alive = false;
    auto die = [&](int count_slot, int weight_slot) {
        if (lead) {
            atomicAdd(&S.ledger[L_STEPS], (unsigned long long)ph.iter);
            kill(S, ph, alive, count_slot, weight_slot);
        }
        alive = false;
    };
    int slot = D, layer = -1;  // next draw of the batch; the layer its step lengths and angles are for
    uint4 r[kTailDraws];
#pragma unroll
    for (int j = 0; j < kTailDraws; ++j) r[j] = make_uint4(0u, 0u, 0u, 0u);
    for (;;) {
        __syncwarp();  // lanes that branched off (tallies, groups at a surface) would each go on alone
        if (!alive && !done) {
            // ---- this group's next photon ----
            int cancelled = 0;
            if (lead) {
                if (P.tail_direct && P.cancel && *P.cancel) cancelled = 1;
                if (!cancelled && !dealt)
                    next = n_groups + (P.tail_direct ? atomicAdd(P.counter, 1ull) : (unsigned long long)atomicAdd(P.tail_next, 1u));
            }
            cancelled = __shfl_sync(gm, cancelled, 0, G);
            next = __shfl_sync(gm, next, 0, G);
            dealt = false;
            done = cancelled || next >= n_next;
            if (cancelled && lead) atomicOr(P.status, 2);
        }
        if (__all_sync(FULL, done)) break;
        if (done) continue;
        if (!alive) {
            if (P.tail_direct) {
                unsigned long long idx = next;
                ph.rdet = -1;
                if (P.mode == 1) {
                    const unsigned long long e = P.replay_list[idx];
                    idx = e >> 16;
                    ph.rdet = (int)(e & 0xffffu);
                }
                launch_photon(P, ph, P.first_id + idx);
                xrow = (blockIdx.x * kTailThreads + threadIdx.x) / G;
                xn = 0;
                if (lead) atomicAdd(&S.ledger[L_LAUNCHED], 1ull);
            } else {
                const TailPhoton& T = P.tail[next];
                ph.px = T.px; ph.py = T.py; ph.pz = T.pz;
                ph.dx = T.dx; ph.dy = T.dy; ph.dz = T.dz;
                ph.time = T.time; ph.trange = T.trange; ph.orange = T.orange; ph.tmin = T.tmin;
                ph.w = (WT)T.w; ph.pid = T.pid;
                ph.layer = T.layer; ph.excl = T.excl; ph.rdet = T.rdet;
                ph.visited = T.visited; ph.iter = T.iter;
                xrow = T.xrow; xn = T.xn;
            }
            find_gap(s_zlo, s_zhi, P.n_zocc, ph.pz, ph.gap_lo, ph.gap_hi);
            if (kLog) ph.rdet = -1;
            alive = true;
            slot = D;
        }
        unsigned* const xl = kLog ? P.xlog + (size_t)xrow * P.xlog_cap : nullptr;
        if (slot == D || layer != ph.layer) {
            if (slot == D) {
#pragma unroll
                for (int j = 0; j < kTailDraws; ++j)
                    r[j] = philox4x32_10(make_uint4((uint32_t)ph.pid, (uint32_t)(ph.pid >> 32), ph.iter + G * j + lane, 0u), P.keys);
                slot = 0;
            }
            layer = ph.layer;
            const DevLayer& L = s_layer[layer];
            __syncwarp(gm);  // every lane has read the previous draws
#pragma unroll
            for (int j = 0; j < kTailDraws; ++j) {
                float4 a;
                float cp = 0.0f;
                a.x = -__logf(u24(r[j].x)) * L.inv_mut;
                if (!kBias) hg_angles(L.hg_a, L.hg_b, L.hg_c, L.hg_d, L.hg_e, u24(r[j].y), u24(r[j].z), a.y, a.z, a.w, cp);
                draw[G * j + lane] = a;
                draw_cp[G * j + lane] = cp;
            }
            __syncwarp(gm);
        }
        // ---- free steps: one short chain each, left by a single branch ----
        if (!kBias) {
            const DevLayer& L = s_layer[layer];
            const bool target = (P.target_mask >> layer) & 1u;
            while (slot < D) {
                const float4 A = draw[slot];
                const float ox = ph.px, oy = ph.py, oz = ph.pz;
                int idx;
                WT dw;
                if (!free_step(P, L, A.x, area_kill, ph, idx, dw)) break;
                if (idx >= 0) {
                    if (lead && dw && P.mode == 0) atomicAdd(&P.absorb[idx], (unsigned long long)dw);
                    absorbed += dw;
                } else {
                    absorbed_out += dw;
                }
                if (target) absorbed_tgt += dw;
                if (!(ph.pz > ph.gap_lo && ph.pz < ph.gap_hi))
                    find_gap(s_zlo, s_zhi, P.n_zocc, ph.pz, ph.gap_lo, ph.gap_hi);
                if (record_planes) {
                    if (lead) cross_planes(P, ox, oy, oz, ph.px, ph.py, ph.pz, ph.w + dw, ph.rdet, xl, xn, n_cross);
                    __syncwarp(gm);
                }
                hg_rotate(A.y, A.z, A.w, draw_cp[slot], ph.dx, ph.dy, ph.dz);
                ++slot;
            }
            if (slot == D) continue;
        }
        // ---- one walk iteration (the transport kernel's) ----
        if (ph.iter >= P.max_steps) {
            budget_hit = 1;
            die(L_N_BUDGET, L_BUDGET);
            continue;
        }
        const int k = slot++;
        const float4 A = draw[k];
        uint4 rk = r[0];
#pragma unroll
        for (int j = 1; j < kTailDraws; ++j)
            if (k / G == j) rk = r[j];
        ph.iter++;
        const DevLayer& L = s_layer[layer];
        Hit hit;
        hit.t = 0.0f;
        hit.tri = -1;
        float step = A.x;
        bool boundary;
        if (L.glass) {
            hit = bvh_nearest(P.nodes, P.tris, P.n_nodes, s_nodes, P.smem_nodes, s_tris, P.smem_tris, ph.px, ph.py, ph.pz,
                              ph.dx, ph.dy, ph.dz, ph.tmin, INFINITY, ph.excl, retests, n_visit, n_tri);
            if (hit.tri < 0) {
                die(L_N_GLASS, L_GLASS);
                continue;
            }
            boundary = true;
        } else {
            const float zend = fmaf(step + kStepExtend, ph.dz, ph.pz);
            if (!in_gap(ph, zend)) {
                if (!(P.grid_nx > 0 && tail_grid_query(P, s_big, s_tris, ph.px, ph.py, ph.pz, ph.dx, ph.dy, ph.dz, ph.tmin,
                                                       step + kStepExtend, ph.excl, hit, retests, n_visit, n_tri)))
                    hit = bvh_nearest(P.nodes, P.tris, P.n_nodes, s_nodes, P.smem_nodes, s_tris, P.smem_tris, ph.px, ph.py,
                                      ph.pz, ph.dx, ph.dy, ph.dz, ph.tmin, step + kStepExtend, ph.excl, retests, n_visit,
                                      n_tri);
            }
            boundary = hit.tri >= 0;
        }
        if (boundary) step = hit.t;
        // move (mcml_kernel.cpp:151-174)
        const float ox = ph.px, oy = ph.py, oz = ph.pz;
        ph.px = fmaf(step, ph.dx, ph.px);
        ph.py = fmaf(step, ph.dy, ph.py);
        ph.pz = fmaf(step, ph.dz, ph.pz);
        if (record_planes && lead) cross_planes(P, ox, oy, oz, ph.px, ph.py, ph.pz, ph.w, ph.rdet, xl, xn, n_cross);
        ph.time = fmaf(step, L.n, ph.time);
        if (!(ph.pz > ph.gap_lo && ph.pz < ph.gap_hi)) find_gap(s_zlo, s_zhi, P.n_zocc, ph.pz, ph.gap_lo, ph.gap_hi);
        if ((P.target_mask >> layer) & 1u) ph.trange += step;
        else ph.orange += step;
        const int idx = area_index(P, ph.px, ph.py, ph.pz, boundary ? 1e-4f : 0.0f);
        if (idx < 0 && area_kill) {
            die(L_N_AREA, L_AREA);
            continue;
        }
        if (boundary) {
            const uint32_t uf = __shfl_sync(gm, L.glass ? rk.x : rk.y, k, G);
            const int crossed = cross_boundary(P, s_layer, s_tris, s_next, L, hit.tri, u24(uf), ph);
            if (crossed == kCrossInvalid) {
                die(L_N_INVALID, L_INVALID);
                continue;
            }
            if (crossed == kCrossLeft) {
                const int det = find_detector(P, s_det, ph);
                if (P.mode == 0) {
                    if (det >= 0) {
                        if (lead) tally_detection(P, S, ph, det);
                        const unsigned n = __shfl_sync(gm, xn, 0, G);
                        if (kLog && n <= P.xlog_cap) {
                            __syncwarp(gm);  // orders the lead lane's log stores before the other lanes' loads
                            for (unsigned j = lane; j < n; j += G) atomicAdd(&P.traj[(size_t)det * P.grid + xl[j]], 1ull);
                            __syncwarp(gm);
                        } else if ((P.flags & XMC_DETECTOR_TRAJ) && lead) {
                            list_for_replay(P, ph.pid, det);
                        }
                    }
                } else if (det != ph.rdet && lead) {
                    atomicAdd(&S.ledger[L_N_REPLAY_MISMATCH], 1ull);
                }
                if (ph.dz < 0.0f) die(L_N_TOP, L_TOP);
                else die(L_N_BOTTOM, L_BOTTOM);
                continue;
            }
        } else {
            // ---- drop (mcml_kernel.cpp:633-642) ----
            WT dw = f2w<WT>(w2f(ph.w) * L.absorb);
            dw = min(dw, ph.w);
            ph.w -= dw;
            if (idx >= 0) {
                if (lead && dw && P.mode == 0) atomicAdd(&P.absorb[idx], (unsigned long long)dw);
                absorbed += dw;
            } else {
                absorbed_out += dw;
            }
            if ((P.target_mask >> layer) & 1u) absorbed_tgt += dw;
            // ---- spin (mcml_kernel.cpp:442-495) ----
            if constexpr (kBias) biased_spin<G>(P, L, layer, ph, bias_gained, bias_lost);
            else hg_rotate(A.y, A.z, A.w, draw_cp[k], ph.dx, ph.dy, ph.dz);
            ph.excl = -1;
            ph.tmin = 0.0f;
        }
        // ---- weight cut / roulette ----
        if (ph.w < P.w_min) {
            if (roulette) {
                const float u = u24(__shfl_sync(gm, L.glass ? rk.y : boundary ? rk.z : rk.w, k, G));
                if (ph.w != 0u && u < P.chance) {
                    const WT nw = min(f2w<WT>(w2f(ph.w) * P.inv_chance), (WT)kWeightOne);
                    if (lead) lat(&S.ledger[L_RGAINED], nw - ph.w);
                    ph.w = nw;
                } else {
                    die(L_N_ROULETTE, L_RKILLED);
                }
            } else {
                die(L_N_CUT, L_CUT);
            }
        }
    }

    // ---- flush: the lead lanes' sums, and every lane's own query counts ----
    if (lead) {
        lat(&S.ledger[L_ABSORBED], absorbed);
        lat(&S.ledger[L_ABSORBED_OUT], absorbed_out);
        lat(&S.ledger[L_ABSORBED_TGT], absorbed_tgt);
        if (kBias) {
            lat(&S.ledger[L_BIAS_GAINED], bias_gained);
            lat(&S.ledger[L_BIAS_LOST], bias_lost);
        }
        if (n_cross) atomicAdd(&S.ledger[L_N_CROSSINGS], (unsigned long long)n_cross);
        if (budget_hit) atomicOr(P.status, 1);
    }
    lat(&S.ledger[L_N_RETEST], retests);
    lat(&S.ledger[L_N_NODES], n_visit);
    lat(&S.ledger[L_N_TRIS], n_tri);
    __syncthreads();
    for (int i = threadIdx.x; i < kLedgerSlots; i += blockDim.x) lat(&P.ledger[i], s_ledger[i]);
    for (int i = threadIdx.x; i < 4 * P.n_dets; i += blockDim.x) lat(&P.det[i], s_dettal[i]);
}

}  // namespace xmc
