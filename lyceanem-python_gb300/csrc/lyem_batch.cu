// lyem_batch.cu -- many scenes x many frequencies, direct + one-bounce paths,
// in one persistent launch.
//
// Each scene is the composition of calculate_scattering_cuda
// (lyceanem/models/frequency_domain.py:195-264) summed over the sources
// (:847-849), evaluated at every frequency of a list:
//   e_p(f)  = sum_n S1_f(n, p)                           scatter excitation
//   E_f(m)  = sum_n S0_f(n, m) + sum_p e_p(f) (.) S2_f(p, m; e_p(f))
// with S_f the per-pair field of em_wave (lyceanem/src/em.cuh:18-120) at
// beta_f and the visibility of raycasting.cuh:19-95, which is the same for
// every frequency and is therefore resolved once.
//
// Work is a queue of items that the warps of a fixed set of resident blocks
// take in order, each warp on its own (no block-wide barrier: a warp whose
// rays end early moves on instead of waiting for the slowest warp of a tile):
//   V items  visibility of one source chunk (32 or 64 sources) against 32
//            sinks, for one of the three stages of a scene (sources ->
//            scatter points, sources -> sinks, scatter points -> sinks): grid
//            DDA, all lanes on the same source at a time, or (sources that are
//            elements) on the same sink; each lane stores its sink's visibility of
//            the chunk as bits of a sink-major mask (one 32-bit word per 32 sources);
//   W items  e_p(f) for a run of (scatter point, frequency group) slots;
//   E items  E_f(m) for a run of (sink, frequency group) slots; both taken 32
//            slots at a time, the lanes of a point sharing its pairs' set-up,
//            or, with few groups, a point at a time, its lanes sharing its
//            sources.
// The queue holds every V item, then every W item, then every E item.  A W
// item needs its scene's sources -> scatter visibility; an E item needs the
// two other visibility stages and all W items of its scene.  They wait on the
// scene's completion counters.  Every item waited on was taken from the queue
// earlier by a running warp that itself waits only on items taken before it,
// so each wait ends; the waits are bounded all the same and raise bit 0 of
// the error word on expiry.
//
// Frequencies: thread (sink, g) of a field item handles the frequencies
// g*FG .. g*FG+FG-1.  The phase beta_f * r of the first one is formed in
// float-float arithmetic (r from the exact coordinate differences, reduced mod
// 2 pi by a Cody-Waite step whose first product-subtraction is exact), and the
// next FG-1 frequencies follow by complex rotation with exp(-j dbeta r), dbeta
// being the uniform frequency step.  FP64 is not used on this path: its rate
// on this GPU is a small fraction of the FP32 rate.  FG = 1 evaluates every
// frequency from its own phase and accepts any frequency list.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <new>
#include <vector>

#include "lyem.h"
#include "lyem_device.cuh"
#include "lyem_internal.cuh"
#include "lyem_walk.cuh"

namespace lyem {
namespace {

constexpr int kBT = 256;  // threads per block (8 independent warps)
constexpr int kWarpSinks = 32;               // sinks of a visibility item (one per lane)
constexpr long long kItemPairs = 1LL << 14;  // pairs of a nominal field item (lyem_batch_items; the queue holds parts)
constexpr int kKinds = 5;
enum Kind { kVisScat = 0, kVisDirect = 1, kVisBounce = 2, kFieldW = 3, kFieldE = 4 };

// The grid fields the walk helpers read (lyem_walk.cuh).
struct GridView {
    const int* cell_start;
    const float4* cell_tris;
    const float4* cell_box;
    float g0[3], g1[3];
    float cell, inv_cell;
    int dims[3];
    float eps;
};

struct DevScene {
    const float* src_pos;
    const float* src_E;
    const float* scat_pos;
    const float* scat_nrm;
    const int* scat_id;
    long long n_src, n_scat;
    GridView grid;
    unsigned int* mask[3];     // sink-major visibility bits of stages kVisScat, kVisDirect, kVisBounce
    long long mask_words[3];   // words per mask row
    float* w;                  // [n_scat][n_freq][6] scatter excitation
    int expect[kKinds];        // items of each kind
    int pad;
};

struct BatchParams {
    const DevScene* scenes;
    const int4* items;  // (kind, scene, a, b)
    int n_items;
    int n_vis;      // V items, the first of the list
    int split;      // parts of a V item (a power of two up to 32): queue positions 0 .. n_vis * split - 1 are its parts
    int turn_all;   // the scatter -> sink items are turned as well
    int n_scenes;
    unsigned int* head;  // queue position
    unsigned int* done;  // [n_scenes][kKinds] finished items
    const float* snk_pos;
    const float* snk_nrm;
    const int* snk_id;
    long long n_snk;
    const float2* beta_ff;  // [n_freq] beta as float-float (hi, lo)
    const float* beta_f;    // [n_freq] beta rounded to FP32
    float2 dbeta_ff;        // uniform frequency step of beta as float-float
    int n_freq;
    int n_groups;           // ceil(n_freq / FG); a field slot is (point, group), slot = point * n_groups + group
    int src_chunk;
    float alpha;
    int skip_diag;
    unsigned int* err;
    unsigned long long* counters;  // [n_scenes][4]: visible pairs of the three stages, ray-triangle tests
    float* field;                  // [n_scenes][n_freq][n_snk][6] output
};

// ---------------------------------------------------------------- queue

// Completion counters.  The walks live on what the SM's L1 holds of the grid, and an acquire (a load of that kind, or
// __threadfence) drops all of it: items end with a release, and a wait polls with relaxed loads, sparingly, and fences
// once at its end.
__device__ __forceinline__ void add_release(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ unsigned ld_relaxed(const unsigned* p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Bounded wait until *ctr >= target; false on expiry.
__device__ bool wait_count(const unsigned* ctr, unsigned target) {
    if (target == 0) return true;
    const long long t0 = clock64();
    unsigned pause = 500;
    while (true) {
        if (ld_relaxed(ctr) >= target) return true;
        if (clock64() - t0 > kWaitCycles) return false;
        __nanosleep(pause);
        pause = min(pause * 2u, 4000u);
    }
}

__device__ bool wait_deps(const BatchParams& P, int kind, int scene) {
    const DevScene& S = P.scenes[scene];
    const unsigned* d = P.done + (long long)scene * kKinds;
    const unsigned parts = (unsigned)P.split;
    bool ok;
    if (kind == kFieldW) {
        ok = wait_count(d + kVisScat, (unsigned)S.expect[kVisScat] * parts);
    } else {
        ok = wait_count(d + kVisDirect, (unsigned)S.expect[kVisDirect] * parts);
        ok = ok && wait_count(d + kVisBounce, (unsigned)S.expect[kVisBounce] * parts);
        ok = ok && wait_count(d + kFieldW, (unsigned)S.expect[kFieldW]);
    }
    __threadfence();
    return ok;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------- V items

// The scene's grid parameters are read from shared memory (filled by the
// caller) rather than held in registers through the walk.
// TURNED: the lanes are 32 of the chunk's sources and the warp walks to one sink of i0 .. i1 - 1 after the other;
// otherwise they are the 32 sinks and it walks from one source after the other.
template <bool CULL, bool TURNED>
__device__ __forceinline__ void vis_walks(const BatchParams& P, const GridView& G, const float* spos, const int* sid, long long n0,
                          int nsrc, const float* kpos, const int* kid, long long m0, long long nk, int i0, int i1,
                          unsigned int* mask, long long words, unsigned int& vis, unsigned int& tests) {
    const int lane = threadIdx.x & 31;
    const bool ok = m0 + lane < nk;
    const int last = TURNED ? (int)min((long long)i1, nk - m0) : 0;
    Walk w;
    for (int g = 0; g < nsrc; g += 32) {
        const long long mine = TURNED ? n0 + g + lane : m0 + lane;  // the lane's point
        const bool has = TURNED ? g + lane < nsrc : ok;
        float lx = 0.f, ly = 0.f, lz = 0.f;
        int id = -1;
        if (has) {
            const float* l = (TURNED ? spos : kpos) + 3 * mine;
            lx = __ldg(l); ly = __ldg(l + 1); lz = __ldg(l + 2);
            const int* ids = TURNED ? sid : kid;
            id = ids ? __ldg(ids + mine) : (int)mine;
        }
        if (!P.skip_diag) id = -1;
        unsigned int word = 0;
        for (int i = TURNED ? i0 : 0; i < (TURNED ? last : min(32, nsrc - g)); ++i) {
            const long long u = TURNED ? m0 + i : n0 + g + i;  // the point all lanes walk to or from
            const int* ids = TURNED ? kid : sid;
            bool hit = !has;
            if (has && id != (ids ? __ldg(ids + u) : (int)u)) {  // (a skipped pair is not tested: visible)
                const float* o = (TURNED ? kpos : spos) + 3 * u;
                const float ux = __ldg(o), uy = __ldg(o + 1), uz = __ldg(o + 2);
                if (TURNED) walk_ray<CULL>(w, lx, ly, lz, ux, uy, uz);
                else walk_ray<CULL>(w, ux, uy, uz, lx, ly, lz);
                if (walk_setup(G, w)) {
                    while (!hit) {
                        while (w.q < w.q1) {
                            ++tests;
                            if (walk_test<CULL>(G, w)) {
                                hit = true;
                                break;
                            }
                        }
                        if (hit || !walk_step(G, w)) break;
                    }
                }
            }
            if (TURNED) {
                const unsigned int b = __ballot_sync(0xffffffffu, !hit);
                if (lane == i) word = b;
            } else {
                __syncwarp();
                if (!hit) word |= 1u << i;
            }
        }
        if (ok && (!TURNED || (lane >= i0 && lane < i1))) {
            mask[(m0 + lane) * words + ((n0 + g) >> 5)] = word;
            vis += __popc(word);
        }
    }
}

template <bool CULL>
__device__ void vis_item(const BatchParams& P, const DevScene& S, const GridView& G, int scene, int stage,
                         long long n0, long long m0, int i0, int i1) {
    const float* spos = stage == kVisBounce ? S.scat_pos : S.src_pos;
    const long long ns = stage == kVisBounce ? S.n_scat : S.n_src;
    const int* sid = stage == kVisBounce ? S.scat_id : nullptr;
    const float* kpos = stage == kVisScat ? S.scat_pos : P.snk_pos;
    const long long nk = stage == kVisScat ? S.n_scat : P.n_snk;
    const int* kid = stage == kVisScat ? S.scat_id : P.snk_id;
    const long long rem = ns - n0;
    const int nsrc = (int)(rem < P.src_chunk ? rem : P.src_chunk);
    unsigned int vis = 0, tests = 0;  // of one lane; diagnostic: wraps only past 2^32 tests
    // The element stages turn the warp round: an array's elements see a sink along rays that cross the same cells (as in
    // grid_transposed_kernel; 8 scenes of up to 3,969 elements, 16 frequencies: 64.0 -> 59.3 ms at (2, 64, 8), 57.1 ->
    // 46.6 at (2, 32, 6)).  Scatter points as sources are turned for few sinks, which lie too far apart to share a walk
    // (the rule of propagation.scatter_schedule), and where items are split.
    if (stage != kVisBounce || P.turn_all)
        vis_walks<CULL, true>(P, G, spos, sid, n0, nsrc, kpos, kid, m0, nk, i0, i1, S.mask[stage], S.mask_words[stage], vis, tests);
    else
        vis_walks<CULL, false>(P, G, spos, sid, n0, nsrc, kpos, kid, m0, nk, i0, i1, S.mask[stage], S.mask_words[stage], vis, tests);
    if (P.counters) {
        const unsigned long long v = warp_sum((unsigned long long)vis);
        const unsigned long long t = warp_sum((unsigned long long)tests);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(P.counters + 4LL * scene + stage, v);
            atomicAdd(P.counters + 4LL * scene + 3, t);
        }
    }
}

// ---------------------------------------------------------------- field items

// What a pair o -> (e, normal nrm) contributes at every frequency.
struct PairCommon {
    float v[6];            // direct form: E - (E.d) d of the excitation E; bounce form: direction d
    int n;                 // bounce form: the source's row
    float sc, a_re;        // -(1/2pi) (n.d) exp(-alpha r) / r, -alpha - 1/r
    float rh, rl;          // path length r in float-float
    float zre, zim;        // exp(-j dbeta r), the rotation of one frequency step
};

template <int FG, bool BOUNCE>
__device__ __forceinline__ PairCommon pair_common(const BatchParams& P, const float* spos, const float* src_E,
                                                  long long n, float ex, float ey, float ez, float nx, float ny,
                                                  float nz) {
    PairCommon c;
    const float* so = spos + 3 * n;
    const float ox = __ldg(so), oy = __ldg(so + 1), oz = __ldg(so + 2);
    const Ray r = make_ray(ox, oy, oz, ex, ey, ez);
    const float inv_r = 1.0f / r.len;
    const float mag = expf(-P.alpha * r.len) * inv_r;
    c.a_re = -P.alpha - inv_r;
    const float nd = nx * r.dx + ny * r.dy + nz * r.dz;
    c.sc = -0.15915494309189535f * nd * mag;
    ff_length(ox, oy, oz, ex, ey, ez, c.rh, c.rl);
    c.zre = 1.f;
    c.zim = 0.f;
    if (FG > 1) {
        // with what the FP32 rounding of the phase drops: the rotation multiplies that of the step up to FG - 1 times
        float zs, zc, rem;
        const float dph = ff_phase_parts(P.dbeta_ff.x, P.dbeta_ff.y, c.rh, c.rl, rem);
        sincos_parts(dph, rem, &zs, &zc);
        c.zre = zc;
        c.zim = -zs;
    }
    c.n = (int)n;
    if (BOUNCE) {
        c.v[0] = r.dx; c.v[1] = r.dy; c.v[2] = r.dz;
        c.v[3] = c.v[4] = c.v[5] = 0.f;
    } else {
        const float2* e2 = reinterpret_cast<const float2*>(src_E + 6 * n);
        const float2 e0 = __ldg(e2), e1 = __ldg(e2 + 1), e3 = __ldg(e2 + 2);
        const float ed_re = e0.x * r.dx + e1.x * r.dy + e3.x * r.dz;
        const float ed_im = e0.y * r.dx + e1.y * r.dy + e3.y * r.dz;
        c.v[0] = e0.x - ed_re * r.dx; c.v[1] = e0.y - ed_im * r.dx;
        c.v[2] = e1.x - ed_re * r.dy; c.v[3] = e1.y - ed_im * r.dy;
        c.v[4] = e3.x - ed_re * r.dz; c.v[5] = e3.y - ed_im * r.dz;
    }
    return c;
}

// The values a lane set up, through shared memory: three float4 a lane.
template <bool BOUNCE>
__device__ __forceinline__ void put_pair(float4 (*ent)[32], int lane, const PairCommon& c) {
    ent[0][lane] = make_float4(c.v[0], c.v[1], c.v[2], c.sc);
    ent[1][lane] = make_float4(BOUNCE ? __int_as_float(c.n) : c.v[3], c.v[4], c.v[5], c.a_re);
    ent[2][lane] = make_float4(c.rh, c.rl, c.zre, c.zim);
}

template <bool BOUNCE>
__device__ __forceinline__ PairCommon get_pair(const float4 (*ent)[32], int lane) {
    const float4 a = ent[0][lane], b = ent[1][lane], d = ent[2][lane];
    PairCommon c;
    c.v[0] = a.x; c.v[1] = a.y; c.v[2] = a.z; c.v[3] = b.x; c.v[4] = b.y; c.v[5] = b.z;
    c.n = BOUNCE ? __float_as_int(b.x) : 0;
    c.sc = a.w; c.a_re = b.w;
    c.rh = d.x; c.rl = d.y; c.zre = d.z; c.zim = d.w;
    return c;
}

// Adds the pair at frequencies f0 .. f0+cnt-1 to acc.
// Bounce form: excitation and weight e_p(f) read from row n of w.
template <int FG, bool BOUNCE>
__device__ __forceinline__ void pair_freqs(const BatchParams& P, const PairCommon& c, const float* w, float2 b0, int f0,
                                           int cnt, float (&acc)[6 * FG]) {
    float sn, cs, rem;
    const float ph = ff_phase_parts(b0.x, b0.y, c.rh, c.rl, rem);
    sincos_parts(ph, rem, &sn, &cs);
    float cre = c.sc * cs, cim = -c.sc * sn;  // sc exp(-j beta_f0 r)
    const float* wrow = BOUNCE ? w + ((long long)c.n * P.n_freq + f0) * 6 : nullptr;
#pragma unroll
    for (int j = 0; j < FG; ++j) {
        if (j < cnt) {
            const float b = __ldg(P.beta_f + f0 + j);
            // loss = (a_re - j beta) * c
            const float lre = c.a_re * cre + b * cim;
            const float lim = c.a_re * cim - b * cre;
            if (!BOUNCE) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    acc[6 * j + 2 * k] += c.v[2 * k] * lre - c.v[2 * k + 1] * lim;
                    acc[6 * j + 2 * k + 1] += c.v[2 * k] * lim + c.v[2 * k + 1] * lre;
                }
            } else {
                const float2 w0 = *reinterpret_cast<const float2*>(wrow + 6 * j);
                const float2 w1 = *reinterpret_cast<const float2*>(wrow + 6 * j + 2);
                const float2 w2 = *reinterpret_cast<const float2*>(wrow + 6 * j + 4);
                const float e[6] = {w0.x, w0.y, w1.x, w1.y, w2.x, w2.y};
                const float ed_re = e[0] * c.v[0] + e[2] * c.v[1] + e[4] * c.v[2];
                const float ed_im = e[1] * c.v[0] + e[3] * c.v[1] + e[5] * c.v[2];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float pr = e[2 * k] - ed_re * c.v[k], pi = e[2 * k + 1] - ed_im * c.v[k];
                    const float tr = pr * lre - pi * lim, ti = pr * lim + pi * lre;  // S2 component
                    acc[6 * j + 2 * k] += e[2 * k] * tr - e[2 * k + 1] * ti;      // weighted by e_p
                    acc[6 * j + 2 * k + 1] += e[2 * k] * ti + e[2 * k + 1] * tr;
                }
            }
            const float nre = cre * c.zre - cim * c.zim;
            cim = cre * c.zim + cim * c.zre;
            cre = nre;
        }
    }
}

// How the lanes of a warp set up the pairs of its sinks (field_item).  A pair's direction, distance, amplitude and
// transverse excitation are the same at every frequency, and cost about as much as three frequencies: `per` pairs of
// each of the warp's sinks are set up at a time, a pair a lane, and every lane of the sink then adds them at its own
// frequencies.  This lane sets up number `rank` of a sink whose bits lane `at` holds, and reads those of its own sink
// from the lanes `from` .. `from` + per - 1.  8 scenes, 1e8 pairs, one frequency a lane, 8 / 16 / 64 frequencies: each
// lane its own pairs 46 / 56 / 134 ms, shared 28.9 / 29.8 / 35.5 ms.
struct Share {
    int per, rank, at, from;
    bool sets;
};

// Sums the pairs of one stage into the thread's accumulator in shared memory
// (sacc[k * kBT + tid], k < 6 FG): per 32 sources in registers, then added.
// Called by all lanes of a warp; ok: the lane has a sink.  (x, y, z) and normal:
// the sink whose pairs the lane sets up.
template <int FG, bool BOUNCE>
__device__ __forceinline__ void field_stage(const BatchParams& P, const unsigned int* row, long long words,
                                            const float* spos, const float* src_E, const float* w, bool ok, float ex,
                                            float ey, float ez, float nx, float ny, float nz, float2 b0, int f0,
                                            int cnt, const Share& sh, float4 (*ent)[32], float* sacc) {
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x;
    for (long long wi = 0; wi < words; ++wi) {
        unsigned int bits = ok ? row[wi] : 0u;
        if (!__any_sync(full, bits != 0)) continue;
        float acc[6 * FG];
#pragma unroll
        for (int k = 0; k < 6 * FG; ++k) acc[k] = 0.f;
        do {
            unsigned int mine = __shfl_sync(full, bits, sh.at);  // without its `rank` lowest bits
            for (int k = 0; k < sh.rank; ++k) mine &= mine - 1;
            const int j = mine ? __ffs(mine) - 1 : 0;
            if (sh.sets && mine)
                put_pair<BOUNCE>(ent, tid & 31, pair_common<FG, BOUNCE>(P, spos, src_E, (wi << 5) + j, ex, ey, ez, nx, ny, nz));
            const int take = min(__popc(bits), sh.per);
            __syncwarp();
            for (int i = 0; i < take; ++i)
                pair_freqs<FG, BOUNCE>(P, get_pair<BOUNCE>(ent, sh.from + i), w, b0, f0, cnt, acc);
            __syncwarp();
            const int last = __shfl_sync(full, j, sh.from + max(take - 1, 0));
            if (take) bits &= ~((2u << last) - 1u);
        } while (__any_sync(full, bits != 0));
#pragma unroll
        for (int k = 0; k < 6 * FG; ++k) sacc[k * kBT + tid] += acc[k];
    }
}

// One warp's 32 consecutive slots (chunk of the scene's slot list).
template <int FG>
__device__ void field_item(const BatchParams& P, const DevScene& S, int scene, int kind, long long chunk,
                           float4 (*ent)[32], float* sacc) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int G = P.n_groups;
    const bool at_sinks = kind == kFieldE;
    const long long nk = at_sinks ? P.n_snk : S.n_scat;
    const long long slot = chunk * 32 + (tid & 31);
    const long long ms = slot / G;
    const int g = (int)(slot - ms * G);
    const int f0 = g * FG;
    const int cnt = min(FG, P.n_freq - f0);
    const bool ok = ms < nk && cnt > 0;
    const int m0 = __shfl_sync(0xffffffffu, (int)ms, 0), g0 = __shfl_sync(0xffffffffu, g, 0);
    const int sinks = (g0 + 31) / G + 1;
    Share sh;
    sh.per = 32 / sinks;
    const int own = lane / sh.per;
    sh.rank = lane - own * sh.per;
    sh.sets = own < sinks && m0 + own < nk;
    sh.at = sh.sets ? max(own * G - g0, 0) : lane;
    sh.from = ((int)ms - m0) * sh.per;
    const long long ks = (long long)m0 + own;  // the sink whose pairs this lane sets up
#pragma unroll
    for (int k = 0; k < 6 * FG; ++k) sacc[k * kBT + tid] = 0.f;
    float ex = 0.f, ey = 0.f, ez = 0.f, nx = 0.f, ny = 0.f, nz = 0.f;
    float2 b0 = make_float2(0.f, 0.f);
    if (ok) b0 = __ldg(P.beta_ff + f0);
    if (sh.sets) {
        const float* kp = (at_sinks ? P.snk_pos : S.scat_pos) + 3 * ks;
        const float* kn = (at_sinks ? P.snk_nrm : S.scat_nrm) + 3 * ks;
        ex = __ldg(kp); ey = __ldg(kp + 1); ez = __ldg(kp + 2);
        nx = __ldg(kn); ny = __ldg(kn + 1); nz = __ldg(kn + 2);
    }
    if (!at_sinks) {
        const long long words = S.mask_words[kVisScat];
        field_stage<FG, false>(P, S.mask[kVisScat] + ms * words, words, S.src_pos, S.src_E, nullptr, ok, ex, ey, ez,
                               nx, ny, nz, b0, f0, cnt, sh, ent, sacc);
        if (ok) {
            float* out = S.w + (ms * P.n_freq + f0) * 6;
            for (int k = 0; k < 6 * cnt; ++k) out[k] = sacc[k * kBT + tid];
        }
        return;
    }
    {
        const long long words = S.mask_words[kVisDirect];
        field_stage<FG, false>(P, S.mask[kVisDirect] + ms * words, words, S.src_pos, S.src_E, nullptr, ok, ex, ey,
                               ez, nx, ny, nz, b0, f0, cnt, sh, ent, sacc);
    }
    if (S.n_scat > 0) {
        const long long words = S.mask_words[kVisBounce];
        field_stage<FG, true>(P, S.mask[kVisBounce] + ms * words, words, S.scat_pos, nullptr, S.w, ok, ex, ey, ez,
                              nx, ny, nz, b0, f0, cnt, sh, ent, sacc);
    }
    if (ok) {
        const long long m = P.snk_id ? (long long)__ldg(P.snk_id + ms) : ms;
        for (int j = 0; j < cnt; ++j) {
            float* out = P.field + (((long long)scene * P.n_freq + f0 + j) * P.n_snk + m) * 6;
#pragma unroll
            for (int k = 0; k < 6; ++k) out[k] = sacc[(6 * j + k) * kBT + tid];
        }
    }
}

// Few frequency groups (kPointGroups at most): a warp takes one point, its lanes a slice of the point's visible sources
// for one group each, every lane with its own pairs; the slices are added at the end.  With a point and group a lane,
// a sink's sources stand one behind the other on one lane, milliseconds for a few thousand of them, while most of the
// chip has nothing to do.  8 scenes, 1e8 pairs, 1 / 4 frequencies (one a lane) 27.4 / 30.2 -> 20.4 / 22.3 ms, 16
// frequencies (four a lane) 41 -> 25.6; 32 frequencies (four a lane, 8 groups) 38.4 -> 32.1; with 16 groups 27.9 -> 33.3.
constexpr int kPointGroups = 8;

// Adds the pairs of one stage: the visible sources' indices are listed (list: 64 ints of the warp) and taken L at a time,
// 16 times in registers, then added to the thread's accumulator (sums in two levels, as in field_stage: one running sum
// of a sink's thousands of pairs was 3 times further off).
template <int FG, bool BOUNCE>
__device__ __forceinline__ void point_stage(const BatchParams& P, const unsigned int* row, long long words,
                                            const float* spos, const float* src_E, const float* w, float ex, float ey,
                                            float ez, float nx, float ny, float nz, float2 b0, int f0, int cnt, int L,
                                            int slice, int* list, float* sacc) {
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned below = (1u << lane) - 1u;
    int held = 0, rounds = 0;
    float acc[6 * FG];
#pragma unroll
    for (int k = 0; k < 6 * FG; ++k) acc[k] = 0.f;
    auto flush = [&]() {
#pragma unroll
        for (int k = 0; k < 6 * FG; ++k) {
            sacc[k * kBT + tid] += acc[k];
            acc[k] = 0.f;
        }
    };
    auto add = [&](int count) {
        if (slice < count) {
            const PairCommon c = pair_common<FG, BOUNCE>(P, spos, src_E, list[slice], ex, ey, ez, nx, ny, nz);
            pair_freqs<FG, BOUNCE>(P, c, w, b0, f0, cnt, acc);
        }
    };
    for (long long w0 = 0; w0 < words; w0 += 32) {
        const unsigned mine = w0 + lane < words ? row[w0 + lane] : 0u;
        unsigned any = __ballot_sync(full, mine != 0);
        while (any) {
            const int k = __ffs(any) - 1;
            any &= any - 1;
            const unsigned bits = __shfl_sync(full, mine, k);
            if ((bits >> lane) & 1u) list[held + __popc(bits & below)] = (int)((w0 + k) << 5) + lane;
            held += __popc(bits);
            __syncwarp();
            while (held >= L) {
                add(L);
                if ((++rounds & 15) == 0) flush();
                const int next = lane < held - L ? list[L + lane] : 0;
                __syncwarp();
                list[lane] = next;
                held -= L;
                __syncwarp();
            }
        }
    }
    add(held);
    flush();
    __syncwarp();
}

template <int FG>
__device__ void point_item(const BatchParams& P, const DevScene& S, int scene, int kind, long long point, int* list,
                           float* sacc) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const bool at_sinks = kind == kFieldE;
    const int G = P.n_groups;
    const int L = G == 1 ? 32 : G == 2 ? 16 : G <= 4 ? 8 : 4;  // slices, a power of two with G L <= 32
    const int slice = lane / G < L ? lane / G : 64;  // (64: a lane left over)
    const int g = lane % G;
    const int f0 = g * FG;
    const int cnt = min(FG, P.n_freq - f0);
    const float* kp = (at_sinks ? P.snk_pos : S.scat_pos) + 3 * point;
    const float* kn = (at_sinks ? P.snk_nrm : S.scat_nrm) + 3 * point;
    const float ex = __ldg(kp), ey = __ldg(kp + 1), ez = __ldg(kp + 2);
    const float nx = __ldg(kn), ny = __ldg(kn + 1), nz = __ldg(kn + 2);
    const float2 b0 = __ldg(P.beta_ff + f0);
#pragma unroll
    for (int k = 0; k < 6 * FG; ++k) sacc[k * kBT + threadIdx.x] = 0.f;
    const int vis = at_sinks ? kVisDirect : kVisScat;
    point_stage<FG, false>(P, S.mask[vis] + point * S.mask_words[vis], S.mask_words[vis], S.src_pos, S.src_E, nullptr, ex,
                           ey, ez, nx, ny, nz, b0, f0, cnt, L, slice, list, sacc);
    if (at_sinks && S.n_scat > 0)
        point_stage<FG, true>(P, S.mask[kVisBounce] + point * S.mask_words[kVisBounce], S.mask_words[kVisBounce],
                              S.scat_pos, nullptr, S.w, ex, ey, ez, nx, ny, nz, b0, f0, cnt, L, slice, list, sacc);
    float acc[6 * FG];
#pragma unroll
    for (int k = 0; k < 6 * FG; ++k) acc[k] = sacc[k * kBT + threadIdx.x];
    for (int o = L / 2; o > 0; o /= 2) {
#pragma unroll
        for (int k = 0; k < 6 * FG; ++k) acc[k] += __shfl_down_sync(full, acc[k], o * G);
    }
    if (slice == 0) {
        const long long m = !at_sinks ? point : P.snk_id ? (long long)__ldg(P.snk_id + point) : point;
#pragma unroll
        for (int j = 0; j < FG; ++j) {
            if (j >= cnt) break;
            float* out = at_sinks ? P.field + (((long long)scene * P.n_freq + f0 + j) * P.n_snk + m) * 6
                                  : S.w + (point * P.n_freq + f0 + j) * 6;
#pragma unroll
            for (int k = 0; k < 6; ++k) out[k] = acc[6 * j + k];
        }
    }
}

// ---------------------------------------------------------------- kernel

// MINB: blocks per SM the register allocation is capped for (1: uncapped).
// Each warp works on its own: lane 0 takes the next queue position while the
// warp works on the current item (the atomic's latency is hidden), so a warp
// holds one taken-but-unstarted item.  Progress still holds: the smallest
// unfinished queue position is always being worked on (its holder took it
// after every item it could be busy with), and it waits only on smaller
// positions, which are finished.
template <bool CULL, int FG, int MINB>
__global__ void __launch_bounds__(kBT, MINB) batch_kernel(const BatchParams P) {
    extern __shared__ float sacc[];
    __shared__ GridView s_grid[kBT / 32];
    __shared__ float4 s_ent[kBT / 32][3][32];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned nxt = 0;
    if (lane == 0) nxt = atomicAdd(P.head, 1u);
    while (true) {
        int kind = -1, scene = 0, a = 0, b = 0, run = 1, part = 0;
        if (lane == 0) {
            unsigned i = nxt;
            const unsigned parts = (unsigned)P.n_vis * (unsigned)P.split;
            if (i < parts) {
                part = (int)(i & (unsigned)(P.split - 1));
                i /= (unsigned)P.split;
            } else {
                i -= parts - (unsigned)P.n_vis;
            }
            if (i < (unsigned)P.n_items) {
                const int4 it = P.items[i];
                kind = it.x;
                scene = it.y;
                a = it.z;
                b = it.w;
                nxt = atomicAdd(P.head, 1u);
                if (kind >= kFieldW && !wait_deps(P, kind, scene)) {
                    atomicOr(P.err, 1u);
                    run = 0;  // the item is skipped; its outputs are not valid
                }
                if (kind < kFieldW) s_grid[wid] = P.scenes[scene].grid;
            }
        }
        kind = __shfl_sync(full, kind, 0);
        scene = __shfl_sync(full, scene, 0);
        a = __shfl_sync(full, a, 0);
        b = __shfl_sync(full, b, 0);
        run = __shfl_sync(full, run, 0);
        part = __shfl_sync(full, part, 0);
        __syncwarp();  // s_grid[wid] is visible to the warp
        if (kind < 0) break;
        if (run) {
            const DevScene& S = P.scenes[scene];
            if (kind < kFieldW)
                vis_item<CULL>(P, S, s_grid[wid], scene, kind, (long long)a, (long long)b,
                               part * (kWarpSinks / P.split), (part + 1) * (kWarpSinks / P.split));
            else if (P.n_groups <= kPointGroups)
                for (int t = 0; t < b; ++t)  // b consecutive points
                    point_item<FG>(P, S, scene, kind, (long long)a + t, reinterpret_cast<int*>(s_ent[wid]), sacc);
            else
                for (int t = 0; t < b; ++t)  // b consecutive 32-slot chunks
                    field_item<FG>(P, S, scene, kind, (long long)a + t, s_ent[wid], sacc);
        }
        __syncwarp();
        if (lane == 0) add_release(P.done + (long long)scene * kKinds + kind, 1u);
    }
}

// ---------------------------------------------------------------- host plan

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct Plan {
    std::vector<int4> items;  // (only where the list is asked for: it can have many millions of entries)
    long long n_vis = 0, n_items = 0;
    std::vector<size_t> off_mask[3], off_w;
    std::vector<int> expect;  // [n_scenes][kKinds]
    long long count[kKinds] = {};  // items of each kind (items holds the field items' parts)
    size_t off_ctrl = 0, ctrl_bytes = 0, off_scenes = 0, off_items = 0, off_beta = 0, off_betaf = 0, total = 0;
};

bool config_ok(const lyem_batch_config* c) {
    if (!c) return false;
    if (!(c->freq_group == 1 || c->freq_group == 2 || c->freq_group == 4 || c->freq_group == 8)) return false;
    if (!(c->src_chunk == 32 || c->src_chunk == 64)) return false;
    if (c->blocks_per_sm < 0 || c->blocks_per_sm > 8) return false;
    if (!(c->eps >= 0.f) || !isfinite(c->eps) || !isfinite(c->alpha)) return false;
    return true;
}

// Workspace layout, numbers of items and, if `list` is set, the items; a pure function of the sizes and the configuration.
// (The list has to be made once, by lyem_batch_prepare.  Making it for each launch and query too: 1,024 elements, 20,000
// scatter points, 16,471 sinks 1.1 ms each.)
int make_plan(const lyem_batch_scene* sc, int n_scenes, long long n_snk, int n_freq, const lyem_batch_config* cfg,
              Plan& pl, bool list = false) {
    if (!sc || n_scenes <= 0 || n_snk <= 0 || n_freq <= 0 || !config_ok(cfg)) return LYEM_ERR_INVALID;
    if (n_snk >= (1LL << 31) || n_freq > 4096) return LYEM_ERR_OVERFLOW;
    const int FG = cfg->freq_group;
    const long long groups = (n_freq + FG - 1) / FG;
    if ((n_snk * groups + 31) / 32 >= (1LL << 31)) return LYEM_ERR_OVERFLOW;  // 32-slot chunk index in an int
    const long long chunk = cfg->src_chunk;
    size_t off = 0;
    pl.off_ctrl = off;
    pl.ctrl_bytes = align256(sizeof(unsigned) * (1 + (size_t)n_scenes * kKinds));
    off += pl.ctrl_bytes;
    pl.off_scenes = off;
    off += align256(sizeof(DevScene) * (size_t)n_scenes);
    pl.off_beta = off;
    off += align256(sizeof(float2) * (size_t)n_freq);
    pl.off_betaf = off;
    off += align256(sizeof(float) * (size_t)n_freq);
    for (int k = 0; k < 3; ++k) pl.off_mask[k].assign(n_scenes, 0);
    pl.off_w.assign(n_scenes, 0);
    pl.expect.assign((size_t)n_scenes * kKinds, 0);
    // scenes in decreasing order of estimated work, so that the big ones start first
    std::vector<double> cost(n_scenes);
    std::vector<int> order(n_scenes);
    for (int s = 0; s < n_scenes; ++s) {
        const long long N = sc[s].n_src, P = sc[s].n_scat;
        if (N < 0 || P < 0 || N >= (1LL << 31) || P >= (1LL << 31)) return LYEM_ERR_INVALID;
        if (N > 0 && (!sc[s].src_pos || !sc[s].src_E)) return LYEM_ERR_INVALID;
        if (P > 0 && (!sc[s].scat_pos || !sc[s].scat_nrm)) return LYEM_ERR_INVALID;
        if (!sc[s].cell_start || !sc[s].cell_tris || (reinterpret_cast<uintptr_t>(sc[s].cell_tris) & 15u) ||
            !sc[s].cell_box || (reinterpret_cast<uintptr_t>(sc[s].cell_box) & 15u))
            return LYEM_ERR_INVALID;
        long long nc = 1;
        for (int k = 0; k < 3; ++k) {
            if (sc[s].grid_dims[k] < 1 || !isfinite(sc[s].grid_origin[k])) return LYEM_ERR_INVALID;
            nc *= sc[s].grid_dims[k];
        }
        if (!(sc[s].grid_cell > 0.f) || !isfinite(sc[s].grid_cell) || nc >= (1LL << 30)) return LYEM_ERR_INVALID;
        if ((P * groups + 31) / 32 >= (1LL << 31)) return LYEM_ERR_OVERFLOW;
        cost[s] = (double)N * (double)n_snk + (double)N * (double)P + (double)P * (double)n_snk;
        order[s] = s;
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[a] > cost[b]; });
    for (int s = 0; s < n_scenes; ++s) {
        const long long N = sc[s].n_src, P = sc[s].n_scat;
        const long long wN = (N + 31) / 32, wP = (P + 31) / 32;
        pl.off_mask[kVisScat][s] = off;
        off += align256(sizeof(unsigned) * (size_t)(P * wN));
        pl.off_mask[kVisDirect][s] = off;
        off += align256(sizeof(unsigned) * (size_t)(n_snk * wN));
        pl.off_mask[kVisBounce][s] = off;
        off += align256(sizeof(unsigned) * (size_t)(n_snk * wP));
        pl.off_w[s] = off;
        off += align256(sizeof(float) * 6 * (size_t)P * (size_t)n_freq);
    }
    pl.items.clear();
    auto add_vis = [&](int s, int stage, long long ns, long long nk) {
        if (list)
            for (long long n0 = 0; n0 < ns; n0 += chunk)
                for (long long t = 0; t < nk; t += kWarpSinks) pl.items.push_back(make_int4(stage, s, (int)n0, (int)t));
        const long long n = ((ns + chunk - 1) / chunk) * ((nk + kWarpSinks - 1) / kWarpSinks);
        pl.expect[(size_t)s * kKinds + stage] = (int)n;
        pl.count[stage] += n;
        pl.n_vis += n;
    };
    for (int s : order) {
        const long long N = sc[s].n_src, P = sc[s].n_scat;
        add_vis(s, kVisScat, N, P);
        add_vis(s, kVisDirect, N, n_snk);
        add_vis(s, kVisBounce, P, n_snk);
    }
    // The nominal field items, which lyem_batch_items reports, are runs of 32-slot
    // chunks (slot = point * groups + group) of about kItemPairs candidate (pair,
    // group) evaluations.  The list holds parts: a chunk each (more where a point has fewer
    // than 64 sources), or a point each (more where it has fewer than 512),
    // since a warp adds their pairs one behind the other whatever the number
    // of groups, and long runs left most warps without work.  8 scenes of up to 178 elements, 1,649 sinks, 8 / 64 frequencies:
    // whole items 9.0 / 25.8 ms, parts 3.4 / 4.4 ms; 8 of up to 4,096, 4,000
    // sinks, 16 / 64 frequencies: 35.6 / 72.8 and 29.8 / 35.3 ms.
    auto add_field = [&](int s, int kind, long long nk, long long pairs_per_sink) {
        const long long chunks = (nk * groups + 31) / 32;
        const long long per_chunk = std::max(1LL, pairs_per_sink * 32 / groups);
        const long long k = std::min(64LL, std::max(1LL, (kItemPairs + per_chunk - 1) / per_chunk));
        pl.count[kind] += (chunks + k - 1) / k;
        const bool by_point = groups <= kPointGroups;  // (point_item: the chunk is a point)
        const long long n = by_point ? nk : chunks;
        const long long part = std::max(1LL, (by_point ? 512 : 64) / std::max(1LL, pairs_per_sink));
        if (list)
            for (long long c = 0; c < n; c += part)
                pl.items.push_back(make_int4(kind, s, (int)c, (int)std::min(part, n - c)));
        pl.expect[(size_t)s * kKinds + kind] = (int)((n + part - 1) / part);
        pl.n_items += (n + part - 1) / part;
    };
    for (int s : order) add_field(s, kFieldW, sc[s].n_scat, sc[s].n_src);
    for (int s : order) add_field(s, kFieldE, n_snk, sc[s].n_src + sc[s].n_scat);
    pl.n_items += pl.n_vis;
    if (pl.n_items >= 0x7fffffffLL) return LYEM_ERR_OVERFLOW;
    pl.off_items = off;
    off += align256(sizeof(int4) * (size_t)pl.n_items);
    pl.total = off;
    return LYEM_OK;
}

// beta as float-float, the uniform step, and whether the list is uniform
void beta_tables(const double* beta, int n, std::vector<float2>& ff, std::vector<float>& f32, float2& step,
                 bool& uniform) {
    ff.resize(n);
    f32.resize(n);
    for (int i = 0; i < n; ++i) {
        const float hi = (float)beta[i];
        ff[i] = make_float2(hi, (float)(beta[i] - (double)hi));
        f32[i] = hi;
    }
    const double d = n > 1 ? (beta[n - 1] - beta[0]) / (double)(n - 1) : 0.0;
    const float dh = (float)d;
    step = make_float2(dh, (float)(d - (double)dh));
    double bmax = 0.0, dev = 0.0;
    for (int i = 0; i < n; ++i) {
        bmax = std::max(bmax, fabs(beta[i]));
        dev = std::max(dev, fabs(beta[i] - (beta[0] + d * (double)i)));
    }
    uniform = dev <= 1e-12 * std::max(bmax, 1.0);
}

template <bool CULL, int FG, int MINB>
cudaError_t launch_batch_t(BatchParams P, int blocks_per_sm, cudaStream_t stream, int* blocks_out) {
    auto kern = batch_kernel<CULL, FG, MINB>;
    const size_t smem = sizeof(float) * 6 * FG * kBT;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int fit = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, kern, kBT, smem);
    if (e != cudaSuccess) return e;
    const int per_sm = blocks_per_sm > 0 ? std::min(blocks_per_sm, std::max(fit, 1)) : std::max(fit, 1);
    const int sms = device_sm_count();
    if (sms <= 0) return cudaErrorInvalidDevice;
    // A V item is 32 or 64 walks (or twice that, turned) one behind the other: the items are split into parts until there
    // are four for every resident warp.  At (2, 64, 8): 2 scenes of up to 64 elements, 500 sinks, 1 frequency 3.12 -> 1.52
    // ms; 4 of up to 986, 673 sinks, 1 frequency 6.54 -> 2.49; 2 of up to 300, 4,000 sinks, 3 frequencies 24.4 -> 16.7; 8 of
    // up to 3,969, 4,000 sinks, 16 frequencies 57.2 -> 52.5 (one part a warp 55.9, 16 parts 50.8).
    const long long want = (long long)per_sm * sms * (kBT / 32) * 4;
    P.split = 1;
    while (P.split < kWarpSinks && (long long)P.n_vis * P.split < want) P.split *= 2;
    P.turn_all = P.split > 1 || P.n_snk <= 2048;
    const int blocks = (int)std::max(1LL, std::min<long long>((long long)per_sm * sms, P.n_items + (long long)P.n_vis * (P.split - 1)));
    kern<<<blocks, kBT, smem, stream>>>(P);
    note_launches(1);
    if (blocks_out) *blocks_out = blocks;
    return cudaGetLastError();
}

template <bool CULL>
cudaError_t launch_batch_c(const BatchParams& P, int fg, int bps, cudaStream_t s, int* b) {
    // register-capped variants: 8 (32 registers) or 4 blocks per SM for up
    // to 4 frequencies per thread, also 6 (40 registers) for 2, 3 for 4 and 8;
    // other requests run the uncapped variant.  Eight blocks at 4 frequencies
    // run the 40-register variant: their 36 KB of shared memory each leave room
    // for six (4 scenes of 1,024 elements, 2,000 scatter points, 4,000 sinks, 16
    // frequencies 32.1 -> 25.6 ms).
    switch (fg) {
        case 1:
            if (bps == 8) return launch_batch_t<CULL, 1, 8>(P, bps, s, b);
            return bps == 4 ? launch_batch_t<CULL, 1, 4>(P, bps, s, b) : launch_batch_t<CULL, 1, 1>(P, bps, s, b);
        case 2:
            if (bps == 8) return launch_batch_t<CULL, 2, 8>(P, bps, s, b);
            if (bps == 6) return launch_batch_t<CULL, 2, 6>(P, bps, s, b);
            return bps == 4 ? launch_batch_t<CULL, 2, 4>(P, bps, s, b) : launch_batch_t<CULL, 2, 1>(P, bps, s, b);
        case 4:
            if (bps == 8) return launch_batch_t<CULL, 4, 6>(P, bps, s, b);
            if (bps == 4) return launch_batch_t<CULL, 4, 4>(P, bps, s, b);
            if (bps == 3) return launch_batch_t<CULL, 4, 3>(P, bps, s, b);
            return launch_batch_t<CULL, 4, 1>(P, bps, s, b);
        default: return bps == 3 ? launch_batch_t<CULL, 8, 3>(P, bps, s, b) : launch_batch_t<CULL, 8, 1>(P, bps, s, b);
    }
}

int fail(cudaError_t e) {
    record_cuda_error(e);
    return e == cudaErrorMemoryAllocation ? LYEM_ERR_NOMEM : LYEM_ERR_CUDA;
}

}  // namespace
}  // namespace lyem

using namespace lyem;

extern "C" {

LYEM_API size_t lyem_batch_workspace(const lyem_batch_scene* scenes, int32_t n_scenes, int64_t n_snk,
                                     int32_t n_freq, const lyem_batch_config* config) {
    Plan pl;
    if (make_plan(scenes, n_scenes, n_snk, n_freq, config, pl) != LYEM_OK) return 0;
    return pl.total;
}

LYEM_API int64_t lyem_batch_items(const lyem_batch_scene* scenes, int32_t n_scenes, int64_t n_snk, int32_t n_freq,
                                  const lyem_batch_config* config, int64_t* per_kind5) {
    Plan pl;
    const int st = make_plan(scenes, n_scenes, n_snk, n_freq, config, pl);
    if (st != LYEM_OK) return -(int64_t)st;
    int64_t total = 0;
    for (int k = 0; k < kKinds; ++k) {
        if (per_kind5) per_kind5[k] = pl.count[k];
        total += pl.count[k];
    }
    return total;
}

LYEM_API int lyem_batch_prepare(const lyem_batch_scene* scenes, int32_t n_scenes, int64_t n_snk,
                                const double* beta, int32_t n_freq, const lyem_batch_config* config, void* d_ws,
                                size_t ws_bytes, void* stream) {
    Plan pl;
    int st = make_plan(scenes, n_scenes, n_snk, n_freq, config, pl);
    if (st != LYEM_OK) return st;
    if (!beta) return LYEM_ERR_INVALID;
    for (int i = 0; i < n_freq; ++i)
        if (!isfinite(beta[i])) return LYEM_ERR_INVALID;
    std::vector<float2> ff;
    std::vector<float> f32;
    float2 step;
    bool uniform;
    beta_tables(beta, n_freq, ff, f32, step, uniform);
    if (config->freq_group > 1 && !uniform) return LYEM_ERR_INVALID;
    if (!d_ws || ws_bytes < pl.total || (reinterpret_cast<uintptr_t>(d_ws) & 255u)) return LYEM_ERR_WORKSPACE;
    try {
        const size_t n = (size_t)pl.n_items;
        pl = Plan();
        pl.items.reserve(n);
        st = make_plan(scenes, n_scenes, n_snk, n_freq, config, pl, true);
    } catch (const std::bad_alloc&) {
        return LYEM_ERR_NOMEM;
    }
    if (st != LYEM_OK) return st;
    char* base = static_cast<char*>(d_ws);
    std::vector<DevScene> ds(n_scenes);
    for (int s = 0; s < n_scenes; ++s) {
        const lyem_batch_scene& c = scenes[s];
        DevScene& d = ds[s];
        memset(&d, 0, sizeof(d));
        d.src_pos = c.src_pos;
        d.src_E = c.src_E;
        d.scat_pos = c.scat_pos;
        d.scat_nrm = c.scat_nrm;
        d.scat_id = c.scat_id;
        d.n_src = c.n_src;
        d.n_scat = c.n_scat;
        d.grid.cell_start = c.cell_start;
        d.grid.cell_tris = reinterpret_cast<const float4*>(c.cell_tris);
        d.grid.cell_box = reinterpret_cast<const float4*>(c.cell_box);
        for (int k = 0; k < 3; ++k) {
            d.grid.g0[k] = c.grid_origin[k];
            d.grid.g1[k] = c.grid_origin[k] + c.grid_dims[k] * c.grid_cell;
            d.grid.dims[k] = c.grid_dims[k];
        }
        d.grid.cell = c.grid_cell;
        d.grid.inv_cell = 1.0f / c.grid_cell;
        d.grid.eps = config->eps;
        const long long wN = (c.n_src + 31) / 32, wP = (c.n_scat + 31) / 32;
        for (int k = 0; k < 3; ++k) d.mask[k] = reinterpret_cast<unsigned int*>(base + pl.off_mask[k][s]);
        d.mask_words[kVisScat] = wN;
        d.mask_words[kVisDirect] = wN;
        d.mask_words[kVisBounce] = wP;
        d.w = reinterpret_cast<float*>(base + pl.off_w[s]);
        for (int k = 0; k < kKinds; ++k) d.expect[k] = pl.expect[(size_t)s * kKinds + k];
    }
    cudaStream_t strm = reinterpret_cast<cudaStream_t>(stream);
    auto put = [&](size_t off, const void* src, size_t bytes) -> cudaError_t {
        if (bytes == 0) return cudaSuccess;
        return cudaMemcpyAsync(base + off, src, bytes, cudaMemcpyHostToDevice, strm);
    };
    cudaError_t e;
    if ((e = put(pl.off_scenes, ds.data(), sizeof(DevScene) * ds.size())) != cudaSuccess) return fail(e);
    if ((e = put(pl.off_items, pl.items.data(), sizeof(int4) * pl.items.size())) != cudaSuccess) return fail(e);
    if ((e = put(pl.off_beta, ff.data(), sizeof(float2) * ff.size())) != cudaSuccess) return fail(e);
    if ((e = put(pl.off_betaf, f32.data(), sizeof(float) * f32.size())) != cudaSuccess) return fail(e);
    // the host tables are released on return: finish the copies first
    if ((e = cudaStreamSynchronize(strm)) != cudaSuccess) return fail(e);
    return LYEM_OK;
}

LYEM_API int lyem_batch_launch(const lyem_batch_scene* scenes, int32_t n_scenes, const float* d_snk_pos,
                               const float* d_snk_nrm, const int32_t* d_snk_id, int64_t n_snk, const double* beta,
                               int32_t n_freq, const lyem_batch_config* config, void* d_ws, size_t ws_bytes,
                               float* d_field_out, uint64_t* d_counters, int32_t* blocks_out, void* stream) {
    Plan pl;
    int st = make_plan(scenes, n_scenes, n_snk, n_freq, config, pl);
    if (st != LYEM_OK) return st;
    if (!beta || !d_snk_pos || !d_snk_nrm || !d_field_out || ((uintptr_t)d_field_out & 7u)) return LYEM_ERR_INVALID;
    if (!d_ws || ws_bytes < pl.total || (reinterpret_cast<uintptr_t>(d_ws) & 255u)) return LYEM_ERR_WORKSPACE;
    std::vector<float2> ff;
    std::vector<float> f32;
    float2 step;
    bool uniform;
    beta_tables(beta, n_freq, ff, f32, step, uniform);
    if (config->freq_group > 1 && !uniform) return LYEM_ERR_INVALID;
    char* base = static_cast<char*>(d_ws);
    cudaStream_t strm = reinterpret_cast<cudaStream_t>(stream);
    BatchParams P;
    memset(&P, 0, sizeof(P));
    P.scenes = reinterpret_cast<const DevScene*>(base + pl.off_scenes);
    P.items = reinterpret_cast<const int4*>(base + pl.off_items);
    P.n_items = (int)pl.n_items;
    P.n_vis = (int)pl.n_vis;
    P.n_scenes = n_scenes;
    P.head = reinterpret_cast<unsigned int*>(base + pl.off_ctrl);
    P.done = P.head + 1;
    P.snk_pos = d_snk_pos;
    P.snk_nrm = d_snk_nrm;
    P.snk_id = d_snk_id;
    P.n_snk = n_snk;
    P.beta_ff = reinterpret_cast<const float2*>(base + pl.off_beta);
    P.beta_f = reinterpret_cast<const float*>(base + pl.off_betaf);
    P.dbeta_ff = step;
    P.n_freq = n_freq;
    P.n_groups = (n_freq + config->freq_group - 1) / config->freq_group;
    P.src_chunk = config->src_chunk;
    P.alpha = (float)config->alpha;
    P.skip_diag = config->self_to_self ? 0 : 1;
    P.err = device_error_word();
    P.counters = reinterpret_cast<unsigned long long*>(d_counters);
    P.field = d_field_out;
    cudaError_t e = cudaMemsetAsync(base + pl.off_ctrl, 0, pl.ctrl_bytes, strm);
    if (e != cudaSuccess) return fail(e);
    if (d_counters) {
        e = cudaMemsetAsync(d_counters, 0, sizeof(uint64_t) * 4 * (size_t)n_scenes, strm);
        if (e != cudaSuccess) return fail(e);
    }
    int blocks = 0;
    e = config->cull ? launch_batch_c<true>(P, config->freq_group, config->blocks_per_sm, strm, &blocks)
                     : launch_batch_c<false>(P, config->freq_group, config->blocks_per_sm, strm, &blocks);
    if (e != cudaSuccess) return fail(e);
    if (blocks_out) *blocks_out = blocks;
    return LYEM_OK;
}

}  // extern "C"
