// lyem_stage.cu -- visibility + fused field kernels ("pair stages").
//
// Thread block = 128 sinks (one per thread) x a chunk of sources.  Each thread
// resolves the visibility of its sink from every source of the chunk, then
// evaluates the field of the visible pairs and sums them over the chunk in
// registers.  Chunk partial sums go to a [n_chunks, n_snk, 6] buffer and a
// second kernel reduces them in FP64 in a fixed order, so results are
// reproducible run to run.  Optionally the kernels also write the per-pair
// network (the reference's output layout) and a visibility bit mask.
//
// Brute force (replaces raycast_brute_force, lyceanem/src/raycasting_brute_force.cuh:68-88):
// triangle tiles of 128 (of 32 in the variant for few triangles) are staged in shared memory by TMA bulk copies
// (double-buffered, mbarrier-completed, bounded waits).  For each source of the chunk a warp takes 32
// triangles at a time, a lane each: it derives the ray-independent part of the test (tvec, qvec, e2.qvec) and drops
// the triangles that face away from the source or that the beam of the warp's 32 rays cannot meet; its rays then test
// the others.  A ray stops at its first hit, and the block stops loading tiles once every ray is resolved.
//
// Grid (replaces raycast_tiles + DDA, lyceanem/src/raycasting_accelerated.cuh:106-268, 458-482):
// each thread walks its segment through a uniform 3-D grid (Amanatides-Woo,
// boundary crossings recomputed from the cell index so no error accumulates)
// and tests the triangles stored contiguously per cell (float4 loads), stopping
// at the first hit.
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>

#include "lyem_device.cuh"
#include "lyem_internal.cuh"
#include "lyem_walk.cuh"

namespace lyem {

__device__ unsigned int g_device_error = 0;

static std::atomic<unsigned long long> g_launches{0};
void note_launches(unsigned long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
unsigned long long launches_so_far() { return g_launches.load(std::memory_order_relaxed); }

// FP32 FMA throughput probe: 8 independent FMA chains per thread.
__global__ void fma_probe_kernel(long long iters, float seed, float* sink) {
    float a0 = seed + threadIdx.x, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f;
    float a4 = a0 + 4.f, a5 = a0 + 5.f, a6 = a0 + 6.f, a7 = a0 + 7.f;
    const float b = 0.999999f, c = 1e-7f;
#pragma unroll 16
    for (long long i = 0; i < iters; ++i) {
        a0 = __fmaf_rn(a0, b, c); a1 = __fmaf_rn(a1, b, c); a2 = __fmaf_rn(a2, b, c); a3 = __fmaf_rn(a3, b, c);
        a4 = __fmaf_rn(a4, b, c); a5 = __fmaf_rn(a5, b, c); a6 = __fmaf_rn(a6, b, c); a7 = __fmaf_rn(a7, b, c);
    }
    float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 12345.f) sink[0] = s;  // keeps the chains alive
}

cudaError_t fma_probe(long long iters, double* fma_per_s, cudaStream_t stream) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    float* sink = nullptr;
    e = cudaMallocAsync(&sink, 16, stream);
    if (e != cudaSuccess) return e;
    cudaEvent_t a, b;
    cudaEventCreate(&a);
    cudaEventCreate(&b);
    const int blocks = sms * 8, threads = 256;
    fma_probe_kernel<<<blocks, threads, 0, stream>>>(iters / 4, 1.f, sink); note_launches(1);
    cudaEventRecord(a, stream);
    fma_probe_kernel<<<blocks, threads, 0, stream>>>(iters, 1.f, sink); note_launches(1);
    cudaEventRecord(b, stream);
    e = cudaEventSynchronize(b);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    cudaFreeAsync(sink, stream);
    if (e != cudaSuccess) return e;
    *fma_per_s = (double)blocks * threads * 8.0 * (double)iters / (ms * 1e-3);
    return cudaGetLastError();
}

int device_sm_count() {
    constexpr int kMaxDev = 64;
    static std::atomic<int> cache[kMaxDev];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    if (dev >= 0 && dev < kMaxDev) {
        const int c = cache[dev].load(std::memory_order_relaxed);
        if (c > 0) return c;
    }
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) return 1;
    if (dev >= 0 && dev < kMaxDev) cache[dev].store(n, std::memory_order_relaxed);
    return n;
}

unsigned capped_blocks(long long n, int threads, int per_sm) {
    long long b = (n + threads - 1) / threads;
    const long long cap = (long long)device_sm_count() * per_sm;
    if (b > cap) b = cap;
    return (unsigned)(b < 1 ? 1 : b);
}

unsigned int* device_error_word() {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_device_error) != cudaSuccess) return nullptr;
    return static_cast<unsigned int*>(p);
}

cudaError_t read_clear_device_errors(unsigned int* flags, cudaStream_t stream) {
    unsigned int zero = 0;
    cudaError_t e = cudaMemcpyFromSymbolAsync(flags, g_device_error, sizeof(unsigned int), 0,
                                              cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyToSymbolAsync(g_device_error, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, stream);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(stream);
}

constexpr int kThreads = 128;
// Brute-force triangle tile (a power of two; two block barriers a tile): 32 / 64 / 128 / 256 / 512 triangles measured
// 0.270 / 0.256 / 0.240 / 0.275 / 0.327 ms on the 8 x 8-array direct scene.
constexpr int kTile = 128;
// Triangles from which on the variant with beams runs.  Below, a ray tests them all as they lie in shared memory: a beam
// costs about as much as a dozen tests.  1,024 sources to 16,471 sinks without / with beams 0.455 / 0.523 ms at 2 triangles,
// 0.747 / 0.774 at 8, 0.796 / 0.770 at 16; two-sided 0.774 / 0.811 at 8, 0.828 / 0.872 at 20, 0.909 / 0.876 at 24.  64 to
// 1,000,000 at 2 triangles 1.47 / 1.83.
constexpr int kBeamTris = 16, kBeamTrisTwoSided = 24;
constexpr int kFewTile = 32;  // tile of the variant without beams: all of its triangles
constexpr int kBruteMaxChunk = 32;  // one bit per source in a 32-bit mask
constexpr int kGridMaxChunk = 64;   // one bit per source in a 64-bit mask

int stage_block_threads() { return kThreads; }
int brute_max_src_chunk() { return kBruteMaxChunk; }
int grid_max_src_chunk() { return kGridMaxChunk; }
int transposed_src_chunk() { return 32; }

template <bool BEAMS>
struct BruteSmem {
    static constexpr int kTris = BEAMS ? kTile : kFewTile;
    float4 raw[2][kTris * 3];
    TriPre pre[BEAMS ? kThreads / 32 : 1][BEAMS ? 32 : 1];  // a warp's candidates of the current 32 triangles
    unsigned long long mbar[2];
};

__device__ __forceinline__ void load_E(const float* base, long long n, float* E) {
    const float2* p = reinterpret_cast<const float2*>(base + 6 * n);
    float2 a = p[0], b = p[1], c = p[2];
    E[0] = a.x; E[1] = a.y; E[2] = b.x; E[3] = b.y; E[4] = c.x; E[5] = c.y;
}

// Field epilogue for one (n, m) pair shared by both kernels.
template <bool WEIGHTED, bool PAIR_OUT>
__device__ __forceinline__ void pair_epilogue(const StageParams& p, long long n, long long m, bool m_ok, bool vis,
                                              float ox, float oy, float oz, float ex, float ey, float ez, float nx,
                                              float ny, float nz, float* acc) {
    if (vis) {
        Ray r = make_ray(ox, oy, oz, ex, ey, ez);
        double rl = path_length_fp64(ox, oy, oz, ex, ey, ez, r.len);
        float E[6], out[6];
        load_E(p.src_E, n, E);
        pair_field(r, rl, E, nx, ny, nz, p.alpha, p.beta_f, p.beta_d, out);
        if (PAIR_OUT) {
            float2* po = reinterpret_cast<float2*>(p.pair_out + 6 * (n * p.n_snk + m));
            po[0] = make_float2(out[0], out[1]);
            po[1] = make_float2(out[2], out[3]);
            po[2] = make_float2(out[4], out[5]);
        }
        if (WEIGHTED) {
            float W[6];
            load_E(p.src_W, n, W);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                acc[2 * k] += W[2 * k] * out[2 * k] - W[2 * k + 1] * out[2 * k + 1];
                acc[2 * k + 1] += W[2 * k] * out[2 * k + 1] + W[2 * k + 1] * out[2 * k];
            }
        } else {
#pragma unroll
            for (int k = 0; k < 6; ++k) acc[k] += out[k];
        }
    } else if (PAIR_OUT && m_ok) {
        float2* po = reinterpret_cast<float2*>(p.pair_out + 6 * (n * p.n_snk + m));
        po[0] = po[1] = po[2] = make_float2(0.f, 0.f);
    }
}

// Mask bits of the warp's 32 sinks for source n, and the per-source visible count.
// ms is the lane's sink slot (m = ms in natural order); lanes past the last
// sink have vis == false.
template <bool MASK_OUT>
__device__ __forceinline__ void record_visibility(const StageParams& p, long long n, long long m, long long ms,
                                                  bool vis) {
    if (!MASK_OUT && !p.src_visible) return;
    unsigned b = __ballot_sync(0xffffffffu, vis);
    if (MASK_OUT && p.snk_order) {
        // permuted sinks: the warp's lanes are not 32 consecutive sinks (mask zeroed by the host)
        if (vis) atomicOr(p.mask_bits + n * p.mask_words + (m >> 5), 1u << (m & 31));
    }
    if ((threadIdx.x & 31) == 0) {
        // natural order: the warp's slots ms .. ms + 31 are the sinks of word ms / 32
        const long long w = ms >> 5;
        if (MASK_OUT && !p.snk_order && w < p.mask_words) p.mask_bits[n * p.mask_words + w] = b;
        if (p.src_visible && b) atomicAdd(p.src_visible + n, __popc(b));
    }
}

__device__ __forceinline__ void flush_block(const StageParams& p, long long m, bool m_ok, const float* acc,
                                            unsigned long long vis_count, unsigned long long tests) {
    if (m_ok) {
        float2* dst = reinterpret_cast<float2*>(p.partial + 6 * ((p.chunk_base + (long long)blockIdx.y) * p.n_snk + m));
        dst[0] = make_float2(acc[0], acc[1]);
        dst[1] = make_float2(acc[2], acc[3]);
        dst[2] = make_float2(acc[4], acc[5]);
        if (p.snk_visible && vis_count) atomicAdd(p.snk_visible + m, (int)vis_count);
    }
    if (p.counters) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            vis_count += __shfl_down_sync(0xffffffffu, vis_count, o);
            tests += __shfl_down_sync(0xffffffffu, tests, o);
        }
        if ((threadIdx.x & 31) == 0) {
            if (vis_count) atomicAdd(p.counters + 0, vis_count);
            if (tests) atomicAdd(p.counters + 1, tests);
        }
    }
}

// The warp's rays from one source as a beam: directions are multiples of (1, sy, sz) in the axes (x, y, z) = (k, k + 1,
// k + 2 mod 3) with x mirrored by `sign`, sy in [y0, y1], sz in [z0, z1]; they end before x = far.
struct BruteBeam {
    int k;  // -1: rays too far apart, no beam
    float sign, y0, y1, z0, z1, far;
};

__device__ __forceinline__ float axis_of(int k, float x, float y, float z) { return k == 0 ? x : k == 1 ? y : z; }

__device__ __forceinline__ float redux_min(float v) {
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float redux_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Beam of the rays of the lanes with `open` (at least one).  A ray without a direction (coincident or non-finite end
// points) hits nothing and is left out.
__device__ __forceinline__ BruteBeam brute_beam(const Ray& r, bool open) {
    const unsigned full = 0xffffffffu;
    BruteBeam b;
    open = open && r.dx * r.dx + r.dy * r.dy + r.dz * r.dz > 0.5f;
    const unsigned who = __ballot_sync(full, open);
    // the axis that the rays' common part is longest along
    const float ax = fmaxf(redux_min(open ? r.dx : 2.f), -redux_max(open ? r.dx : -2.f));
    const float ay = fmaxf(redux_min(open ? r.dy : 2.f), -redux_max(open ? r.dy : -2.f));
    const float az = fmaxf(redux_min(open ? r.dz : 2.f), -redux_max(open ? r.dz : -2.f));
    const float m = fmaxf(ax, fmaxf(ay, az));
    b.k = -1;
    if (!who || !(m > 0.15f)) return b;
    b.k = ax == m ? 0 : ay == m ? 1 : 2;
    const int lead = __ffs(who) - 1;
    b.sign = copysignf(1.f, __shfl_sync(full, axis_of(b.k, r.dx, r.dy, r.dz), lead));
    const float x = axis_of(b.k, r.dx, r.dy, r.dz) * b.sign, inv = 1.f / x;
    const float sy = axis_of(b.k, r.dy, r.dz, r.dx) * inv, sz = axis_of(b.k, r.dz, r.dx, r.dy) * inv;
    const float y = __shfl_sync(full, sy, lead), z = __shfl_sync(full, sz, lead);
    // widened by far more than the rounding of the slopes
    b.y0 = redux_min(open ? sy : y) - 0x1p-16f;
    b.y1 = redux_max(open ? sy : y) + 0x1p-16f;
    b.z0 = redux_min(open ? sz : z) - 0x1p-16f;
    b.z1 = redux_max(open ? sz : z) + 0x1p-16f;
    b.far = redux_max(open ? r.len * x : 0.f) * 1.001f;
    return b;
}

// Whether no ray of the beam from o can hit the triangle.  With t = o - v0 the test's numerators are linear in the ray
// direction D: u = D.(e2 x t), v = D.(t x e1), A = D.(e2 x e1), and w = -t.(e2 x e1).  A hit has u, v, A - u - v >= 0 and
// 0 < w < A len (two-sided: all by A's sign) to within FP32 rounding, so the triangle is missed when one of them fails
// over the whole slope rectangle by more than `slack`: the rounding of the test's and of this evaluation, for
// directions scaled to x = 1, is below 2^-19 (1 + |sy| + |sz|) times the product of the vectors' 1-norms.
template <bool CULL>
__device__ __forceinline__ bool beam_misses(const BruteBeam& B, const TriPre& p) {
    const int k = B.k;
    const float tx = axis_of(k, p.b.z, p.b.w, p.c.x), ty = axis_of(k, p.b.w, p.c.x, p.b.z), tz = axis_of(k, p.c.x, p.b.z, p.b.w);
    const float ax = axis_of(k, p.a.x, p.a.y, p.a.z), ay = axis_of(k, p.a.y, p.a.z, p.a.x), az = axis_of(k, p.a.z, p.a.x, p.a.y);
    const float bx = axis_of(k, p.a.w, p.b.x, p.b.y), by = axis_of(k, p.b.x, p.b.y, p.a.w), bz = axis_of(k, p.b.y, p.a.w, p.b.x);
    const float na = fabsf(ax) + fabsf(ay) + fabsf(az), nb = fabsf(bx) + fabsf(by) + fabsf(bz);
    const float nt = fabsf(tx) + fabsf(ty) + fabsf(tz);
    const float smax = fmaxf(fabsf(B.y0), fabsf(B.y1)) + fmaxf(fabsf(B.z0), fabsf(B.z1));
    const float slack = (0x1p-19f + 0x1p-19f * smax) * (nt + na) * (na + nb);
    // gradients of u, v and A (cyclic axes keep the cross products), x mirrored with the beam
    float ux = (by * tz - bz * ty) * B.sign, uy = bz * tx - bx * tz, uz = bx * ty - by * tx;
    float vx = (ty * az - tz * ay) * B.sign, vy = tz * ax - tx * az, vz = tx * ay - ty * ax;
    const float nx = by * az - bz * ay;
    float cx = nx * B.sign, cy = bz * ax - bx * az, cz = bx * ay - by * ax;
    float w = -(tx * nx + ty * cy + tz * cz);
    const float ym = 0.5f * (B.y0 + B.y1), zm = 0.5f * (B.z0 + B.z1), yh = B.y1 - ym, zh = B.z1 - zm;
    float am = cx + ym * cy + zm * cz;
    const float ah = yh * fabsf(cy) + zh * fabsf(cz) + slack;
    if (!CULL) {  // the sign of A has to be the same over the beam
        const float s = am < 0.f ? -1.f : 1.f;
        am = fabsf(am);
        if (!(am > ah)) return false;
        ux *= s; uy *= s; uz *= s;
        vx *= s; vy *= s; vz *= s;
        cx *= s; cy *= s; cz *= s;
        w *= s;
    }
    cx -= ux + vx; cy -= uy + vy; cz -= uz + vz;
    const float amax = am + ah, ws = slack * nt;
    return amax < 0.f || w < -ws || w > amax * B.far + ws ||
           ux + ym * uy + zm * uz + yh * fabsf(uy) + zh * fabsf(uz) < -slack ||
           vx + ym * vy + zm * vz + yh * fabsf(vy) + zh * fabsf(vz) < -slack ||
           cx + ym * cy + zm * cz + yh * fabsf(cy) + zh * fabsf(cz) < -slack;
}

// Registers capped so that 9 blocks fit an SM: the 8 x 8-array direct scene's 1,344 blocks then run in one wave on 152
// SMs.  Bound by the FP32 work of the per-triangle part, which every warp does for its own beam (about 180 instructions per 32
// triangles).  Against tests of every triangle by every ray: 64 sources, 2,664 sinks, 1,024 triangles 0.279 -> 0.240 ms
// with the sinks in their natural order, 0.161 in direction order (two-sided test 0.620 -> 0.447 / 0.277); 256 sources,
// 16,380 sinks 3.89 -> 1.67 / 1.23.
template <bool CULL, bool WEIGHTED, bool PAIR_OUT, bool MASK_OUT, bool BEAMS>
__global__ void __launch_bounds__(kThreads, 9) brute_stage_kernel(const StageParams p) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    constexpr int kTris = BruteSmem<BEAMS>::kTris;
    BruteSmem<BEAMS>& sm = *reinterpret_cast<BruteSmem<BEAMS>*>(smem_raw);

    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31;
    const long long ms = (long long)blockIdx.x * kThreads + tid;
    const bool m_ok = ms < p.n_snk;
    const long long m = m_ok ? (p.snk_order ? (long long)p.snk_order[ms] : ms) : 0;
    const long long n0 = (p.chunk_base + (long long)blockIdx.y) * p.src_chunk;
    const long long rem = p.n_src - n0;
    const int nsrc = (int)(rem < p.src_chunk ? rem : p.src_chunk);
    auto src_index = [&](int s) -> long long {
        return p.src_order ? (long long)p.src_order[n0 + s] : n0 + s;
    };

    float ex = 0.f, ey = 0.f, ez = 0.f;
    if (m_ok) {
        ex = p.snk_pos[3 * m]; ey = p.snk_pos[3 * m + 1]; ez = p.snk_pos[3 * m + 2];
    }
    uint32_t pending = 0, blocked = 0;
    for (int s = 0; s < nsrc; ++s)
        if (m_ok && !(p.skip_diag && src_index(s) == m)) pending |= 1u << s;

    const long long T = p.n_tris;
    const int ntiles = (int)((T + kTris - 1) / kTris);
    const uint32_t mb0 = smem_addr(&sm.mbar[0]), mb1 = smem_addr(&sm.mbar[1]);
    if (tid == 0) {
        mbar_init(mb0, 1);
        mbar_init(mb1, 1);
        fence_mbar_init();
    }
    __syncthreads();
    auto issue = [&](int k) {
        long long first = (long long)k * kTris;
        long long cnt = T - first < kTris ? T - first : kTris;
        tma_load_1d(smem_addr(&sm.raw[k & 1][0]), p.tris + 3 * first, (uint32_t)(cnt * 48), (k & 1) ? mb1 : mb0);
    };
    int issued = ntiles < 2 ? ntiles : 2;
    if (tid == 0)
        for (int k = 0; k < issued; ++k) issue(k);

    unsigned long long tests = 0;
    bool timed_out = false;
    // with one source per block (the automatic shape for few sources) the lane's
    // ray and the warp's beam are formed once instead of once per tile
    Ray r1 = Ray{0.f, 0.f, 0.f, 0.f};
    BruteBeam b1;
    b1.k = -1;
    if (nsrc == 1) {
        const float* so = p.src_pos + 3 * src_index(0);
        r1 = vis_ray<CULL>(so[0], so[1], so[2], ex, ey, ez);
        if (BEAMS) b1 = brute_beam(r1, pending & 1u);
    }
    TriPre* pre = sm.pre[BEAMS ? tid >> 5 : 0];
    int k = 0;
    for (; k < ntiles; ++k) {
        if (!__syncthreads_or(pending != 0)) break;
        // the vote is a barrier: tile k - 1 has been read by every thread, and its buffer takes tile k + 1
        if (k >= 1 && issued == k + 1 && issued < ntiles) {
            if (tid == 0) {
                fence_proxy_async_smem();
                issue(issued);
            }
            ++issued;
        }
        bool ok = mbar_wait_bounded((k & 1) ? mb1 : mb0, (k >> 1) & 1, kWaitCycles);
        if (__syncthreads_or(!ok)) { timed_out = true; break; }
        const int cnt = (int)(T - (long long)k * kTris < kTris ? T - (long long)k * kTris : kTris);
        const float4* rt = sm.raw[k & 1];
        for (int s = 0; s < nsrc; ++s) {
            bool open = (pending >> s) & 1u;
            if (!__any_sync(full, open)) continue;
            const float* so = p.src_pos + 3 * src_index(s);
            const float ox = so[0], oy = so[1], oz = so[2];
            Ray r = r1;
            BruteBeam beam = b1;
            if (nsrc > 1) {
                r = vis_ray<CULL>(ox, oy, oz, ex, ey, ez);
                if (BEAMS) beam = brute_beam(r, open);
            }
            if (!BEAMS && open) {
                int j = 0;
                while (j < cnt && !hit_full<CULL>(r, ox, oy, oz, rt[3 * j], rt[3 * j + 1], rt[3 * j + 2], p.eps)) ++j;
                open = j == cnt;
                tests += open ? cnt : j + 1;
            }
            for (int base = 0; BEAMS && base < cnt; base += 32) {
                const int j = base + lane;
                bool keep = j < cnt;
                if (keep) {
                    const TriPre t = make_tripre(ox, oy, oz, rt[3 * j], rt[3 * j + 1], rt[3 * j + 2]);
                    // culling test: w = e2.qvec not positive is a miss for every ray, bit for bit (cull_tail)
                    if (CULL) keep = t.d.x > 0.f;
                    if (keep && beam.k >= 0) keep = !beam_misses<CULL>(beam, t);
                    if (keep) pre[lane] = t;
                }
                unsigned cand = __ballot_sync(full, keep);
                __syncwarp();
                while (cand) {
                    const int c = __ffs(cand) - 1;
                    cand &= cand - 1;
                    if (open && hit_pre<CULL>(r, pre[c], p.eps)) {
                        open = false;
                        tests += c + 1;  // (a dropped triangle counts as tested: the ray's outcome is decided)
                    }
                }
                if (open) tests += cnt - base < 32 ? cnt - base : 32;
                if (!__any_sync(full, open)) break;
                __syncwarp();
            }
            if (!open && ((pending >> s) & 1u)) {
                pending &= ~(1u << s);
                blocked |= 1u << s;
            }
            __syncwarp();
        }
    }
    // Wait (bounded) for copies still in flight before the block may exit.
    for (int j = k; j < issued; ++j) {
        if (timed_out && j == k) continue;
        if (!mbar_wait_bounded((j & 1) ? mb1 : mb0, (j >> 1) & 1, kWaitCycles)) timed_out = true;
    }
    if (timed_out) {
        if (tid == 0) atomicOr(&g_device_error, 1u);
        return;
    }

    float nx = 0.f, ny = 0.f, nz = 0.f;
    if (m_ok) {
        nx = p.snk_nrm[3 * m]; ny = p.snk_nrm[3 * m + 1]; nz = p.snk_nrm[3 * m + 2];
    }
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    unsigned long long vis_count = 0;
    for (int s = 0; s < nsrc; ++s) {
        const long long n = src_index(s);
        const bool vis = m_ok && !((blocked >> s) & 1u);
        record_visibility<MASK_OUT>(p, n, m, ms, vis);
        const float* so = p.src_pos + 3 * n;
        pair_epilogue<WEIGHTED, PAIR_OUT>(p, n, m, m_ok, vis, so[0], so[1], so[2], ex, ey, ez, nx, ny, nz, acc);
        vis_count += vis;
    }
    flush_block(p, m, m_ok, acc, vis_count, tests);
}

// Grid stage.  Each lane owns one sink and resolves the rays from the chunk's
// sources to it.  A ray walks the uniform grid (Amanatides-Woo; the boundary
// crossings are recomputed from the cell index, so no error accumulates) and
// tests the triangles stored contiguously per cell (float4 loads), stopping at
// its first hit.  Two schedules of the rays over the lanes:
//   lockstep  all lanes of a warp trace source s, then source s + 1, ...; ray
//             set-up runs in lockstep, a warp waits for its longest ray;
//   refill    each lane moves to its next source when its ray ends, but new
//             rays are started in batches (once `refill_lanes` lanes of the
//             warp are idle, or none is busy) so the set-up code is not
//             serialised lane by lane.
// Visibility of the chunk is kept as a 64-bit blocked mask; the field epilogue
// then takes each lane from one of its own visible sources to the next, or, with
// a per-pair output, all lanes through the sources in lockstep.
constexpr int kLockstep = 0;
constexpr int kRefill = 1;
// Lockstep with the registers capped so that 10, 12 or 16 blocks of 128
// threads fit an SM.  More resident warps hide more of the triangle-load
// latency: on the 28 GHz one-bounce scene the scatter->sink stage takes 1357 ms
// uncapped (60 registers, 8 blocks), 1184 / 1067 / 969 ms capped at 10 / 12 /
// 16 blocks, the last with some spilling; 16 is the default schedule.
constexpr int kLockstep10 = 2;
constexpr int kLockstep12 = 3;
constexpr int kLockstep16 = 4;
// Two phases (registers capped for 16 or 12 blocks per SM).  Phase 1 runs the
// lockstep schedule but walks each ray only up to parameter near_dist (most
// blocked rays end near their origin: the own-surface triangle, local
// clutter); the rays still open there are appended, source-major, to a queue
// of the warp in shared memory (ballot + prefix count).  Phase 2 takes them 32
// at a time, each lane one ray (the sink coordinates come from the owning lane
// by shuffle), and walks them from near_dist to their end, so the lanes of a
// warp hold live rays of one or two sources instead of idling behind the
// longest ray of each source.
constexpr int kTwoPhase16 = 5;
constexpr int kTwoPhase12 = 6;
// kLockstep16 for a launch that p.choice may turn off (a variant of its own: the test costs the walk a register).
constexpr int kChosen16 = 7;

// COUNT = false (only with the default schedule, when the caller asks for no
// counters) leaves the per-test counting out of the walk: one instruction and
// one register less in the innermost loop (scatter->sink stage of the 28 GHz
// scene 448 -> 440 ms).
template <bool CULL, bool WEIGHTED, bool PAIR_OUT, bool MASK_OUT, int MODE, bool COUNT = true>
__global__ void __launch_bounds__(kThreads, MODE == kLockstep10 ? 10 : (MODE == kLockstep12 || MODE == kTwoPhase12) ? 12 : (MODE == kLockstep16 || MODE == kChosen16 || MODE == kTwoPhase16) ? 16 : 1) grid_stage_kernel(const StageParams p) {
    if (MODE == kChosen16 && *p.choice != p.choice_is) return;
    // 32-bit indices (fewer live registers in the walk): the entry point keeps
    // n_src and n_snk below 2^31 - 256
    const int tid = threadIdx.x;
    const int ms = (int)blockIdx.x * kThreads + tid;
    const bool m_ok = ms < p.n_snk;
    const int m = m_ok ? (p.snk_order ? p.snk_order[ms] : ms) : 0;
    const int n0 = (int)((p.chunk_base + (long long)blockIdx.y) * p.src_chunk);
    const int rem = (int)p.n_src - n0;
    const int nsrc = rem < p.src_chunk ? rem : p.src_chunk;
    auto src_index = [&](int s) -> int {
        return p.src_order ? p.src_order[n0 + s] : n0 + s;
    };
    float ex = 0.f, ey = 0.f, ez = 0.f;
    if (m_ok) {
        ex = p.snk_pos[3 * (long long)m]; ey = p.snk_pos[3 * (long long)m + 1]; ez = p.snk_pos[3 * (long long)m + 2];
    }
    unsigned long long blocked = 0;
    unsigned int tests = 0;  // diagnostic count of one lane (64 rays at most); wraps only past 2^32 tests
    Walk w;
    if (MODE == kTwoPhase16 || MODE == kTwoPhase12) {
        __shared__ int s_hint[kGridMaxChunk];
        __shared__ unsigned long long s_blk[kThreads / 32][32];
        extern __shared__ unsigned short s_queue[];  // per warp: src_chunk x 32 entries (source << 5 | lane)
        const int lane = tid & 31, warp = tid >> 5;
        unsigned short* queue = s_queue + (size_t)warp * p.src_chunk * 32;
        s_blk[warp][lane] = 0ull;
        for (int s = warp; s < nsrc; s += kThreads / 32) {
            const float* so = p.src_pos + 3 * (long long)src_index(s);
            const int h = warp_nearest_ref(p, so[0], so[1], so[2]);
            if (lane == 0) s_hint[s] = h;
        }
        __syncthreads();
        const float near = p.near_dist;
        const unsigned full = 0xffffffffu;
        int count = 0;  // the same in every lane of the warp
        for (int s = 0; s < nsrc; ++s) {
            const int n = src_index(s);
            bool far = false;
            if (m_ok && !(p.skip_diag && n == m)) {
                const float* so = p.src_pos + 3 * (long long)n;
                walk_ray<CULL>(w, so[0], so[1], so[2], ex, ey, ez);
                const int hint = s_hint[s];
                bool hit = false;
                if (hint >= 0) {
                    ++tests;
                    hit = walk_test_ref<CULL>(p, w, hint);
                }
                if (!hit && walk_setup(p, w)) {
                    while (true) {
                        while (w.q < w.q1) {
                            ++tests;
                            if (walk_test<CULL>(p, w)) { hit = true; break; }
                        }
                        if (hit) break;
                        const int st = walk_step_until(p, w, near);
                        if (st != 1) {
                            far = st == 2;
                            break;
                        }
                    }
                }
                if (hit) blocked |= 1ull << s;
            }
            const unsigned fb = __ballot_sync(full, far);
            if (far) queue[count + __popc(fb & ((1u << lane) - 1u))] = (unsigned short)((s << 5) | lane);
            count += __popc(fb);
        }
        __syncwarp();
        for (int base = 0; base < count; base += 32) {
            const int i = base + lane;
            const bool has = i < count;
            const unsigned e = has ? queue[i] : 0u;
            const int owner = (int)(e & 31u), s = (int)(e >> 5);
            const float qx = __shfl_sync(full, ex, owner), qy = __shfl_sync(full, ey, owner),
                        qz = __shfl_sync(full, ez, owner);
            if (has) {
                const float* so = p.src_pos + 3 * (long long)src_index(s);
                walk_ray<CULL>(w, so[0], so[1], so[2], qx, qy, qz);
                bool hit = false;
                if (walk_setup_from(p, w, near)) {
                    while (!hit) {
                        while (w.q < w.q1) {
                            ++tests;
                            if (walk_test<CULL>(p, w)) { hit = true; break; }
                        }
                        if (hit || !walk_step(p, w)) break;
                    }
                }
                if (hit) atomicOr(&s_blk[warp][owner], 1ull << s);
            }
        }
        __syncwarp();
        blocked |= s_blk[warp][lane];
    } else if (MODE != kRefill) {
        // per source of the chunk, the triangle nearest to it (one warp per source):
        // tried first by every ray from that source
        __shared__ int s_hint[kGridMaxChunk];
        for (int s = tid >> 5; s < nsrc; s += kThreads / 32) {
            const float* so = p.src_pos + 3 * (long long)src_index(s);
            const int h = warp_nearest_ref(p, so[0], so[1], so[2]);
            if ((tid & 31) == 0) s_hint[s] = h;
        }
        __syncthreads();
        for (int s = 0; s < nsrc; ++s) {
            const int n = src_index(s);
            if (!m_ok || (p.skip_diag && n == m)) continue;
            const float* so = p.src_pos + 3 * (long long)n;
            walk_ray<CULL>(w, so[0], so[1], so[2], ex, ey, ez);
            const int hint = s_hint[s];
            bool hit = false;
            if (hint >= 0) {  // a hit on any triangle blocks the segment, walked or not
                if (COUNT) ++tests;
                hit = walk_test_ref<CULL>(p, w, hint);
            }
            if (!hit && !walk_setup(p, w)) continue;
            while (!hit) {
                while (w.q < w.q1) {
                    if (COUNT) ++tests;
                    if (walk_test<CULL>(p, w)) { hit = true; break; }
                }
                if (hit || !walk_step(p, w)) break;
            }
            if (hit) blocked |= 1ull << s;
        }
    } else {
        int s = -1;
        bool has = false;
        // next source of this lane that needs a walk (untested and off-grid rays are visible)
        auto refill = [&]() {
            while (++s < nsrc) {
                const int n = src_index(s);
                if (p.skip_diag && n == m) continue;
                const float* so = p.src_pos + 3 * (long long)n;
                if (walk_begin<CULL>(p, w, so[0], so[1], so[2], ex, ey, ez)) { has = true; return; }
            }
        };
        const unsigned full = 0xffffffffu;
        while (true) {
            const bool can = !has && m_ok && s + 1 < nsrc;
            const unsigned busy = __ballot_sync(full, has);
            const unsigned idle = __ballot_sync(full, can);
            if (busy == 0 && idle == 0) break;
            if (can && (busy == 0 || __popc(idle) >= p.refill_lanes)) refill();
            if (has) {
                while (w.q < w.q1) {
                    ++tests;
                    if (walk_test<CULL>(p, w)) {
                        blocked |= 1ull << s;
                        has = false;
                        break;
                    }
                }
                if (has && !walk_step(p, w)) has = false;
            }
        }
    }

    float nx = 0.f, ny = 0.f, nz = 0.f;
    if (m_ok) {
        nx = p.snk_nrm[3 * (long long)m]; ny = p.snk_nrm[3 * (long long)m + 1]; nz = p.snk_nrm[3 * (long long)m + 2];
    }
    float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    unsigned long long vis_count = 0;
    if (PAIR_OUT) {
        for (int k = 0; k < nsrc; ++k) {
            const int n = src_index(k);
            const bool vis = m_ok && !((blocked >> k) & 1ull);
            record_visibility<MASK_OUT>(p, n, m, ms, vis);
            const float* so = p.src_pos + 3 * (long long)n;
            pair_epilogue<WEIGHTED, PAIR_OUT>(p, n, m, m_ok, vis, so[0], so[1], so[2], ex, ey, ez, nx, ny, nz, acc);
            vis_count += vis;
        }
    } else {
        // each lane goes from one of its own visible sources to the next: the warp takes as many steps as its
        // busiest sink has visible sources, not as many as sources that any of its sinks sees (28 GHz
        // scatter->sink stage 424.5 -> 416.6 ms)
        if (MASK_OUT || p.src_visible)
            for (int k = 0; k < nsrc; ++k)
                record_visibility<MASK_OUT>(p, src_index(k), m, ms, m_ok && !((blocked >> k) & 1ull));
        unsigned long long seen = m_ok ? ~blocked & (~0ull >> (64 - nsrc)) : 0ull;
        vis_count = __popcll(seen);
        while (seen) {
            const int n = src_index(__ffsll((long long)seen) - 1);
            seen &= seen - 1;
            const float* so = p.src_pos + 3 * (long long)n;
            pair_epilogue<WEIGHTED, PAIR_OUT>(p, n, m, true, true, so[0], so[1], so[2], ex, ey, ez, nx, ny, nz, acc);
        }
    }
    flush_block(p, m, m_ok, acc, vis_count, tests);
}

// Transposed grid stage (traversal 38).  The lanes of a warp are the 32
// sources of the block's chunk, and a warp traces them to one sink after the
// other, so the 32 rays a warp walks together end at the same sink.  When
// the sources are the elements of an array (millimetres apart) those rays cross
// the same cells and test the same triangles, where a warp of the lockstep
// schedule holds 32 directions from one source (a CPU model of the walk on the
// 28 GHz scene: 78.5 instead of 124.8 test iterations per 32 array rays).  The
// field of each sink is summed over the warp's lanes in a fixed butterfly order
// and lane 0 writes the chunk's partial sum of that sink.
//
// A warp takes one to four sinks (transposed_sinks): the walk is bound by
// latency, and a warp per sink gives the most warps and spreads neighbouring sinks,
// whose rays share cells, over the warps of an SM.  256 elements, 120,000 triangles, 32 / 8 / 4 / 2 / 1 sinks a warp:
// to 20,000 scatter points - / 1.05 / 0.91 / 0.85 / 0.81 ms (lockstep 2.08), to 4,186 sinks 1.23 / - / - / - / 0.28
// (0.60); the two array stages of the 28 GHz scene (1,024 elements) 11.3 -> 10.1 and 8.2 -> 7.2 ms.  So few sinks do not pay
// the search for a source's own-surface triangle that the lockstep schedule makes.
constexpr int kTChunk = 32;

// Sinks per warp of the transposed schedule: more than one only where the launch has far more warps than the GPU
// holds (4,096 elements to 65,341 sinks: 33.6 / 33.0 / 32.8 / 34.5 ms with 1 / 2 / 4 / 8).
static int transposed_sinks(long long n_src, long long n_snk) {
    const long long chunks = (n_src + kTChunk - 1) / kTChunk;
    const long long want = (long long)device_sm_count() * 4096;
    int k = 4;
    while (k > 1 && chunks * ((n_snk + k - 1) / k) < want) k /= 2;
    return k;
}

template <bool CULL, bool WEIGHTED, bool PAIR_OUT, bool MASK_OUT, bool COUNT>
__global__ void __launch_bounds__(kThreads, 16) grid_transposed_kernel(const StageParams p) {
    if (p.choice && *p.choice != p.choice_is) return;
    const unsigned full = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long chunk = p.chunk_base + (long long)blockIdx.y;
    const int n0 = (int)(chunk * kTChunk);
    const int nsrc = (int)p.n_src - n0 < kTChunk ? (int)p.n_src - n0 : kTChunk;
    const bool n_ok = lane < nsrc;
    const int n = n_ok ? (p.src_order ? p.src_order[n0 + lane] : n0 + lane) : 0;
    const int spw = p.snk_per_warp;
    float ox = 0.f, oy = 0.f, oz = 0.f;
    if (n_ok) {
        const float* so = p.src_pos + 3 * (long long)n;
        ox = so[0]; oy = so[1]; oz = so[2];
    }
    const int ms0 = ((int)blockIdx.x * (kThreads / 32) + warp) * spw;  // the warp's first sink slot
    unsigned vis_mask = 0;                                    // bit k: this lane's source sees slot ms0 + k
    unsigned int tests = 0;
    Walk w;
    for (int k = 0; k < spw; ++k) {
        const int ms = ms0 + k;
        if (ms >= p.n_snk) break;  // the same in every lane
        const int m = p.snk_order ? p.snk_order[ms] : ms;
        const float ex = p.snk_pos[3 * (long long)m], ey = p.snk_pos[3 * (long long)m + 1],
                    ez = p.snk_pos[3 * (long long)m + 2];
        bool vis = n_ok;  // untested pairs (the skipped diagonal, segments off the grid) are visible
        if (n_ok && !(p.skip_diag && n == m)) {
            bool hit = false;
            if (walk_begin<CULL>(p, w, ox, oy, oz, ex, ey, ez)) {
                while (!hit) {
                    while (w.q < w.q1) {
                        if (COUNT) ++tests;
                        if (walk_test<CULL>(p, w)) { hit = true; break; }
                    }
                    if (hit || !walk_step(p, w)) break;
                }
            }
            vis = !hit;
        }
        if (vis) {
            vis_mask |= 1u << k;
            if (MASK_OUT && p.snk_order) atomicOr(p.mask_bits + (long long)n * p.mask_words + (m >> 5), 1u << (m & 31));
        }
        float acc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const float nx = p.snk_nrm[3 * (long long)m], ny = p.snk_nrm[3 * (long long)m + 1],
                    nz = p.snk_nrm[3 * (long long)m + 2];
        pair_epilogue<WEIGHTED, PAIR_OUT>(p, n, m, n_ok, vis, ox, oy, oz, ex, ey, ez, nx, ny, nz, acc);
#pragma unroll
        for (int c = 0; c < 6; ++c)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(full, acc[c], o);
        const unsigned b = __ballot_sync(full, vis);
        if (lane == 0) {
            float2* dst = reinterpret_cast<float2*>(p.partial + 6 * (chunk * p.n_snk + m));
            dst[0] = make_float2(acc[0], acc[1]);
            dst[1] = make_float2(acc[2], acc[3]);
            dst[2] = make_float2(acc[4], acc[5]);
            if (p.snk_visible && b) atomicAdd(p.snk_visible + m, __popc(b));
        }
    }
    if (n_ok) {
        if (MASK_OUT && !p.snk_order && ms0 < p.n_snk) {
            if (vis_mask)  // (mask zeroed by the host)
                atomicOr(p.mask_bits + (long long)n * p.mask_words + (ms0 >> 5), vis_mask << (ms0 & 31));
        }
        if (p.src_visible && vis_mask) atomicAdd(p.src_visible + n, __popc(vis_mask));
    }
    if (p.counters) {
        unsigned long long v = __popc(vis_mask), t = tests;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            v += __shfl_down_sync(full, v, o);
            t += __shfl_down_sync(full, t, o);
        }
        if (lane == 0) {
            if (v) atomicAdd(p.counters + 0, v);
            if (t) atomicAdd(p.counters + 1, t);
        }
    }
}

// Sums of the chunks' partial sums in FP64: PARTS threads per element, each a run of the chunks, the runs added in order.
// One thread per element leaves the loads of its chunks one behind the other, eight per element leave most of a block
// idle where there are few chunks.
template <int PARTS>
__global__ void __launch_bounds__(256) reduce_partials_kernel(const float* __restrict__ partial, long long n_chunks,
                                                             long long n_elem, float* __restrict__ out, int accumulate,
                                                             const int* __restrict__ choice, long long chosen_chunks) {
    constexpr int kWidth = 256 / PARTS;
    __shared__ double s_part[PARTS][kWidth];
    if (choice && *choice) n_chunks = chosen_chunks;
    const int slot = threadIdx.x % kWidth, part = threadIdx.x / kWidth;
    const long long per = (n_chunks + PARTS - 1) / PARTS;
    const long long c0 = part * per, c1 = c0 + per < n_chunks ? c0 + per : n_chunks;
    for (long long base = (long long)blockIdx.x * kWidth; base < n_elem; base += (long long)gridDim.x * kWidth) {
        const long long i = base + slot;
        double s = PARTS == 1 && accumulate && i < n_elem ? (double)out[i] : 0.0;
        if (i < n_elem) {
#pragma unroll 8
            for (long long c = c0; c < c1; ++c) s += (double)partial[c * n_elem + i];
        }
        if (PARTS > 1) {
            s_part[part][slot] = s;
            __syncthreads();
            if (part == 0 && i < n_elem) {
                s = accumulate ? (double)out[i] : 0.0;
#pragma unroll
                for (int k = 0; k < PARTS; ++k) s += s_part[k][slot];
            }
        }
        if (part == 0 && i < n_elem) out[i] = (float)s;
        if (PARTS > 1) __syncthreads();
    }
}

// Extent of the sources, by one block: 16,384 of them are 200 KB, and the stage that waits for it takes milliseconds.
__global__ void __launch_bounds__(1024) source_choice_kernel(const float* __restrict__ pos, const int* __restrict__ order,
                                                            int n, float cell, int* __restrict__ choice) {
    __shared__ float s_lo[3][32], s_hi[3][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    bool bad = false;
    for (int i = threadIdx.x; i < n; i += 1024) {
        const float* p = pos + 3 * (long long)(order ? order[i] : i);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float v = p[k];
            bad |= !(fabsf(v) < INFINITY);
            lo[k] = fminf(lo[k], v);
            hi[k] = fmaxf(hi[k], v);
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
        if (lane == 0) {
            s_lo[k][warp] = lo[k];
            s_hi[k][warp] = hi[k];
        }
    }
    bad = __syncthreads_or(bad);
    if (threadIdx.x == 0) {
        double d2 = 0.0;
        for (int k = 0; k < 3; ++k) {
            float a = s_lo[k][0], b = s_hi[k][0];
            for (int w = 1; w < 32; ++w) {
                a = fminf(a, s_lo[k][w]);
                b = fmaxf(b, s_hi[k][w]);
            }
            const double e = (double)(b - a);
            d2 += e * e;
        }
        *choice = !bad && sqrt(d2) <= kCompactCells * (double)cell;
    }
}

cudaError_t launch_source_choice(const float* src_pos, const int* src_order, long long n_src, float cell, int* choice,
                                 cudaStream_t stream) {
    source_choice_kernel<<<1, 1024, 0, stream>>>(src_pos, src_order, (int)n_src, cell, choice); note_launches(1);
    return cudaGetLastError();
}

template <bool CULL, bool WEIGHTED, bool PAIR_OUT, bool MASK_OUT>
static cudaError_t launch_t(const StageParams& p0, cudaStream_t stream) {
    const long long chunks = (p0.n_src + p0.src_chunk - 1) / p0.src_chunk;
    const unsigned tiles = (unsigned)((p0.n_snk + kThreads - 1) / kThreads);
    // gridDim.y is limited to 65535: launch the source chunks in slices
    for (long long base = 0; base < chunks; base += 65535) {
        StageParams p = p0;
        p.chunk_base = base;
        dim3 grid(tiles, (unsigned)(chunks - base < 65535 ? chunks - base : 65535));
        if (p.cell_start) {
            if (p.refill_lanes == -116 || p.refill_lanes == -112) {
                const size_t qbytes = (size_t)(kThreads / 32) * p.src_chunk * 32 * sizeof(unsigned short);
                if (p.refill_lanes == -116)
                    grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kTwoPhase16><<<grid, kThreads, qbytes, stream>>>(p);
                else
                    grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kTwoPhase12><<<grid, kThreads, qbytes, stream>>>(p);
            } else if (p.refill_lanes == -38) {
                p.snk_per_warp = transposed_sinks(p.n_src, p.n_snk);
                grid.x = (unsigned)((p.n_snk + p.snk_per_warp * (kThreads / 32) - 1) / (p.snk_per_warp * (kThreads / 32)));
                if (p.counters)
                    grid_transposed_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, true><<<grid, kThreads, 0, stream>>>(p);
                else
                    grid_transposed_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, false><<<grid, kThreads, 0, stream>>>(p);
            } else if (p.refill_lanes == -16 && p.choice) {
                if (p.counters)
                    grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kChosen16><<<grid, kThreads, 0, stream>>>(p);
                else
                    grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kChosen16, false>
                        <<<grid, kThreads, 0, stream>>>(p);
            } else if (p.refill_lanes == -16) {
                if (p.counters)
                    grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kLockstep16><<<grid, kThreads, 0, stream>>>(p);
                else
                    grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kLockstep16, false>
                        <<<grid, kThreads, 0, stream>>>(p);
            }
            else if (p.refill_lanes == -12)
                grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kLockstep12><<<grid, kThreads, 0, stream>>>(p);
            else if (p.refill_lanes == -10)
                grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kLockstep10><<<grid, kThreads, 0, stream>>>(p);
            else if (p.refill_lanes > 0)
                grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kRefill><<<grid, kThreads, 0, stream>>>(p);
            else
                grid_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, kLockstep><<<grid, kThreads, 0, stream>>>(p);
            note_launches(1);
        } else {
            const bool beams = p.n_tris >= (CULL ? kBeamTris : kBeamTrisTwoSided);
            const size_t smem = beams ? sizeof(BruteSmem<true>) : sizeof(BruteSmem<false>);
            auto kern = beams ? brute_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, true>
                              : brute_stage_kernel<CULL, WEIGHTED, PAIR_OUT, MASK_OUT, false>;
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
            kern<<<grid, kThreads, smem, stream>>>(p); note_launches(1);
        }
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <bool CULL, bool WEIGHTED, bool PAIR_OUT>
static cudaError_t launch_m(const StageParams& p, cudaStream_t s) {
    return p.mask_bits ? launch_t<CULL, WEIGHTED, PAIR_OUT, true>(p, s) : launch_t<CULL, WEIGHTED, PAIR_OUT, false>(p, s);
}
template <bool CULL, bool WEIGHTED>
static cudaError_t launch_p(const StageParams& p, cudaStream_t s) {
    return p.pair_out ? launch_m<CULL, WEIGHTED, true>(p, s) : launch_m<CULL, WEIGHTED, false>(p, s);
}
template <bool CULL>
static cudaError_t launch_w(const StageParams& p, cudaStream_t s) {
    return p.src_W ? launch_p<CULL, true>(p, s) : launch_p<CULL, false>(p, s);
}

cudaError_t launch_pair_stage(const StageParams& p, int cull, cudaStream_t stream) {
    if (p.n_src == 0 || p.n_snk == 0) return cudaSuccess;
    return cull ? launch_w<true>(p, stream) : launch_w<false>(p, stream);
}

cudaError_t launch_reduce_partials(const float* partial, long long n_chunks, long long n_snk, float* out,
                                   int accumulate, cudaStream_t stream, const int* choice,
                                   long long chosen_chunks) {
    const long long n_elem = 6 * n_snk;
    if (n_elem == 0) return cudaSuccess;
    // Eight threads per element where one each are too few threads for the chunks' loads: at 1 / 8 / 64 / 512 chunks, us
    // with one and with eight, 15,984 elements 5.7 / 6.4 / 20 / 121 and 5.6 / 5.8 / 10 / 45, 98,826 elements 5.6 / 8.5 /
    // 34 / 230 and 9.8 / 12 / 31 / 198, 392,046 elements 7.7 / 18 / 107 / 813 and 22 / 30 / 105 / 745, 6,000,000 elements
    // 40 / 194 / 1,431 and 217 / 356 / 1,525.
    const long long chunks = n_chunks > chosen_chunks ? n_chunks : chosen_chunks;
    if (n_elem <= 2048 * (chunks > 8 ? chunks : 8))
        reduce_partials_kernel<8><<<capped_blocks(n_elem, 32, 64), 256, 0, stream>>>(partial, n_chunks, n_elem, out,
                                                                                    accumulate, choice, chosen_chunks);
    else
        reduce_partials_kernel<1><<<capped_blocks(n_elem, 256, 16), 256, 0, stream>>>(partial, n_chunks, n_elem, out,
                                                                                     accumulate, choice, chosen_chunks);
    note_launches(1);
    return cudaGetLastError();
}

}  // namespace lyem
