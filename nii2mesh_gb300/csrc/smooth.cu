// smooth.cu — pre-smooth (src/meshify.c:170-216) and the volume reductions of
// meshify (range, bbox; src/meshify.c:305-371).
//
// The blur is three separable 5-tap passes (x, then y, then z) whose every
// tap sum is rounded exactly as the reference's double arithmetic rounds it
// (exact.cuh), so the output is bit-identical to quick_smooth().  One
// streaming kernel per pass (k_pass_x, k_pass_axis): a fast FP32 proof
// decides ~97 % of the taps, the rest are batched per warp and recomputed in
// FP64 by full warps; the z pass also reduces the range (min/max), the count
// of non-finite voxels and the bbox of voxels >= iso.  Traffic: 8 B per voxel
// per pass, three passes.  (The batched atlas smooths its binary
// sub-boxes from their bits instead, atlas.cu.)
#include <float.h>
#include <math.h>
#include <stddef.h>
#include <stdlib.h>

#include <cuda.h>            // CUtensorMap and its enums (the encoder comes from the driver at run time)
#include <cudaTypedefs.h>

#include <algorithm>
#include <map>
#include <mutex>

#include "smooth_core.cuh"

namespace {
using namespace smooth;

// range / bbox / non-finite count of an existing volume: a bounded grid whose
// warps stride over the rows, so the block flushes (one set of atomics each)
// stay few; every reduction is a min, max or count, so the order is free
__global__ void __launch_bounds__(256) k_stats(const float *__restrict__ vol, int nx, int ny, int nz, int z0, float iso,
                                               VolStats *st, bool minmax) {
    grid_wait();
    Acc acc;
    acc.init();
    const long long nrows = (long long)ny * nz;
    const int wpb = blockDim.x >> 5, lane = threadIdx.x & 31;
    for (long long r = (long long)blockIdx.x * wpb + (threadIdx.x >> 5); r < nrows; r += (long long)gridDim.x * wpb) {
        const int z = (int)(r / ny), y = (int)(r - (long long)z * ny);
        const float *row = vol + r * nx;
#pragma unroll 4
        for (int x = lane; x < nx; x += 32) acc.add(__ldg(row + x), x, y, z0 + z, iso);
    }
    acc.flush(st, minmax);
}
}  // namespace

void stats_init_host(VolStats *h) {
    h->vmin = INT_MAX;
    h->vmax = INT_MIN;
    for (int i = 0; i < 3; i++) { h->lo[i] = INT_MAX; h->hi[i] = INT_MIN; }
    h->nonfinite = 0;
    h->masked = 0;
}

// ---- three separable passes with batched exact fix-ups -------------------------
// x pass in -> out, y pass out -> tmp, z pass tmp -> out (with the range and
// bbox reductions).  Each pass evaluates every tap with the fast path; the
// voxels whose rounding the fast path cannot prove (about 2.5 % on data whose
// voxels share an exponent) are staged per warp in shared memory and, 32 at a
// time, recomputed with the reference's double sequence by the full warp, so
// each FP64 instruction serves 32 voxels.  A pass never reads its own
// outputs, so fix-ups can run whenever a batch is full.  Passes run at full
// occupancy with no redundant taps and no block-wide waits.
namespace {
constexpr unsigned FULL = 0xffffffffu;

// The pass being run: input, output, tap stride (1, nx or nx*ny) and, for
// the z pass, the reductions.
struct Pass {
    const float *in;
    float *out;
    unsigned stride;
    int nx, ny;
    unsigned nxy;
    float iso;
    VolStats *st;
};

// Per-warp stack of failed voxels in shared memory (sized by the kernel for
// 31 leftover entries plus what its steps push between drains).  All 32 lanes
// call push, drain and finish together; push adds at most 32 entries, drain
// recomputes full batches of 32.
template <bool STATS>
struct FixStage {
    unsigned *buf;
    int n;   // warp-uniform fill
    __device__ __forceinline__ void run(const Pass &P, Acc &acc, int lo, int cnt, int lane) {
        __syncwarp();
        if (lane < cnt) {
            const unsigned v = buf[lo + lane];
            const float *p = P.in + v;
            const long long s = P.stride;
            const float r = tap5_double(p[-2 * s], p[-s], p[0], p[s], p[2 * s]);
            P.out[v] = r;
            if (STATS) acc.add(r, (int)(v % (unsigned)P.nx), (int)((v / (unsigned)P.nx) % (unsigned)P.ny), (int)(v / P.nxy), P.iso);
        }
        __syncwarp();
    }
    __device__ __forceinline__ void push(bool fail, unsigned vox, int lane) {
        const unsigned m = __ballot_sync(FULL, fail);
        if (fail) buf[n + __popc(m & ((1u << lane) - 1u))] = vox;
        n += __popc(m);
    }
    // every lane queues the voxels base + k * step for the set bits k of fm
    // (one warp scan of the lanes' counts instead of one ballot per output)
    __device__ __forceinline__ void push_mask(unsigned fm, unsigned base, unsigned step, int lane) {
        if (!__any_sync(FULL, fm != 0u)) return;
        const int c = __popc(fm);
        int incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        int at = n + incl - c;
        while (fm) {
            const int k = __ffs(fm) - 1;
            fm &= fm - 1u;
            buf[at++] = base + (unsigned)k * step;
        }
        n += __shfl_sync(FULL, incl, 31);
    }
    __device__ __forceinline__ void drain(const Pass &P, Acc &acc, int lane) {
        while (n >= 32) {
            n -= 32;
            run(P, acc, n, 32, lane);
        }
    }
    __device__ __forceinline__ void finish(const Pass &P, Acc &acc, int lane) {
        drain(P, acc, lane);
        if (n) run(P, acc, 0, n, lane);
        n = 0;
    }
};

// K outputs from the K + 4 inputs w[0 .. K+3] of one lane (output k is the tap
// sum of w[k .. k+4]).  When the K + 4 magnitudes lie within a factor 64 of one
// another the split path decides each tap (exact.cuh: tap5_split), otherwise
// tap5_fast; bit k of the returned mask marks an output neither could decide
// (r[k] is then a placeholder that the FP64 fix-up overwrites).
template <int K>
__device__ __forceinline__ unsigned taps_run(const float (&w)[K + 4], float (&r)[K]) {
    float mx = fabsf(w[0]), mn = fabsf(w[0]);
#pragma unroll
    for (int k = 1; k < K + 4; k++) {
        mx = fmaxf(mx, fabsf(w[k]));
        mn = fminf(mn, fabsf(w[k]));
    }
    unsigned fm = 0;
    if (split_group_ok(mn, mx)) {
        float h[K + 4], l[K + 4];
#pragma unroll
        for (int k = 0; k < K + 4; k++) split12(w[k], h[k], l[k]);
        const float mth = FMUL(mx, 0x1p-8f);
#pragma unroll
        for (int k = 0; k < K; k++) {
            float t;
            if (!tap5_split(h[k], l[k], h[k + 1], l[k + 1], h[k + 2], l[k + 2], h[k + 3], l[k + 3], h[k + 4], l[k + 4],
                            mth, &t))
                fm |= 1u << k;
            r[k] = t;
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; k++) {
            float t = w[k + 2];
            if (!tap5_fast(w[k], w[k + 1], w[k + 2], w[k + 3], w[k + 4], &t)) fm |= 1u << k;
            r[k] = t;
        }
    }
    return fm;
}

// x pass: each warp takes whole rows (rows row0 .. row1-1 of the volume).
__global__ void __launch_bounds__(256) k_pass_x(Pass P, unsigned row0, unsigned row1) {
    grid_wait();
    __shared__ unsigned stage_buf[8][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    FixStage<false> F{stage_buf[w], 0};   // < 32 entries between steps, + 32
    Acc acc;   // unused by the x pass
    const int nx = P.nx;
    const unsigned nwarps = gridDim.x * (blockDim.x / 32);
    for (unsigned row = row0 + blockIdx.x * (blockDim.x / 32) + w; row < row1; row += nwarps) {
        const unsigned r0 = row * (unsigned)nx;
        for (int x0 = 0; x0 < nx; x0 += 32) {
            const int x = x0 + lane;
            const unsigned v = r0 + (unsigned)x;
            bool fail = false;
            if (x < nx) {
                float o;
                if (x >= 2 && x <= nx - 3) {
                    const float *p = P.in + v;
                    fail = !tap5_fast(__ldg(p - 2), __ldg(p - 1), __ldg(p), __ldg(p + 1), __ldg(p + 2), &o);
                } else {
                    o = __ldg(P.in + v);
                }
                if (!fail) P.out[v] = o;
            }
            F.push(fail, v, lane);
            F.drain(P, acc, lane);
        }
    }
    F.finish(P, acc, lane);
}

// x pass for rows whose length is a multiple of 4 (16-byte aligned rows):
// each thread takes 4 consecutive voxels with three float4 loads (its own and
// the neighbours' halves, mostly L1 hits) and one float4 store; voxels whose
// fast path fails are stored as placeholders and fixed by the same warp.
__global__ void __launch_bounds__(256) k_pass_x4(Pass P, unsigned row0, unsigned row1) {
    grid_wait();
    __shared__ unsigned stage_buf[8][32 * 5];   // < 32 between drains, + 4 per lane per step
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    FixStage<false> F{stage_buf[w], 0};
    Acc acc;   // unused by the x pass
    const int nx = P.nx, nq = nx / 4;
    const unsigned nwarps = gridDim.x * (blockDim.x / 32);
    for (unsigned row = row0 + blockIdx.x * (blockDim.x / 32) + w; row < row1; row += nwarps) {
        const float4 *r4 = reinterpret_cast<const float4 *>(P.in + (size_t)row * nx);
        float4 *o4 = reinterpret_cast<float4 *>(P.out + (size_t)row * nx);
        for (int q0 = 0; q0 < nq; q0 += 32) {
            const int q = q0 + lane, x0 = 4 * q;
            const bool act = q < nq;
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 A = act && q > 0 ? __ldg(r4 + q - 1) : zero;
            const float4 B = act ? __ldg(r4 + q) : zero;
            const float4 C = act && q + 1 < nq ? __ldg(r4 + q + 1) : zero;
            // x0-2 .. x0+5; past the row ends (only face voxels read them) stand-ins from
            // this quad, so that the group test of the split path sees row values only
            const float w[8] = {q > 0 ? A.z : B.x, q > 0 ? A.w : B.x, B.x, B.y, B.z, B.w,
                                q + 1 < nq ? C.x : B.w, q + 1 < nq ? C.y : B.w};
            float o[4];
            unsigned fm = 0;
            if (act) {
                fm = taps_run<4>(w, o);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (x0 + j < 2 || x0 + j > nx - 3) {   // face voxels keep their input
                        o[j] = w[2 + j];
                        fm &= ~(1u << j);
                    }
                o4[q] = make_float4(o[0], o[1], o[2], o[3]);
            }
            F.push_mask(fm, row * (unsigned)nx + (unsigned)x0, 1u, lane);
            F.drain(P, acc, lane);
        }
    }
    F.finish(P, acc, lane);
}

// y and z passes: the volume is viewed as (outer, len, inner) with the pass
// axis of length len and stride inner.  A task is SEGS consecutive groups of
// 32 inner positions and a run of K positions along the axis; each lane
// slides a register window along the axis.  STATS: the z pass, which also
// reduces range and bbox.
// Outputs positions [p_lo, p_hi) along the axis of outer slices
// [outer0, outer0 + nouter) (the staged upload runs the passes slab by slab).
template <int K, int SEGS, bool STATS>
__global__ void __launch_bounds__(256, 4) k_pass_axis(Pass P, int len, unsigned outer0, unsigned nouter, int p_lo,
                                                      int p_hi) {
    grid_wait();
    __shared__ unsigned stage_buf[8][32 * (K + 1)];   // < 32 entries between segments, + up to 32 K per segment
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    FixStage<STATS> F{stage_buf[wid], 0};
    const unsigned inner = P.stride;
    const unsigned nseg = (inner + 31) / 32, nchunk = (nseg + SEGS - 1) / SEGS;
    const unsigned nrun = (unsigned)(p_hi - p_lo + K - 1) / K;
    const unsigned ntask = nchunk * nrun * nouter;
    const unsigned nwarps = gridDim.x * (blockDim.x / 32);
    Acc acc;
    acc.init();
    for (unsigned t = blockIdx.x * (blockDim.x / 32) + wid; t < ntask; t += nwarps) {
        const unsigned chunk = t % nchunk, rest = t / nchunk;
        const int p0 = p_lo + (int)(rest % nrun) * K;
        const unsigned o = outer0 + rest / nrun;
        const unsigned sbeg = chunk * SEGS, send = min(sbeg + SEGS, nseg);
        const bool interior = p0 >= 2 && p0 + K <= len - 2 && p0 + K <= p_hi;   // no face rows, whole run inside
        for (unsigned seg = sbeg; seg < send; seg++) {
            const unsigned i = seg * 32 + lane;
            const bool act = i < inner;
            const unsigned base = o * (unsigned)len * inner + i;
            float w[K + 4];
            int gx = 0, gy = 0;
            if (STATS) { gx = (int)(i % (unsigned)P.nx); gy = (int)(i / (unsigned)P.nx); }
            if (interior) {
                const float *q = P.in + base + (unsigned)(p0 - 2) * inner;
#pragma unroll
                for (int k = 0; k < K + 4; k++) w[k] = act ? __ldg(q + (unsigned)k * inner) : 0.f;
                float r[K];
                unsigned fm = 0;
                if (act) {
                    fm = taps_run<K>(w, r);
#pragma unroll
                    for (int k = 0; k < K; k++) P.out[base + (unsigned)(p0 + k) * inner] = r[k];   // placeholder where fm has bit k
                    if (STATS) acc.add_run<K>(r, ~fm, gx, gy, p0, P.iso);
                }
                F.push_mask(fm, base + (unsigned)p0 * inner, inner, lane);
            } else {
#pragma unroll
                for (int k = 0; k < K + 4; k++) {
                    const int pos = p0 - 2 + k;
                    w[k] = (act && pos >= 0 && pos < len) ? __ldg(P.in + base + (unsigned)pos * inner) : 0.f;
                }
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const int pos = p0 + k;
                    bool fail = false;
                    const unsigned v = base + (unsigned)pos * inner;
                    if (act && pos < p_hi) {
                        float r = w[k + 2];
                        if (pos >= 2 && pos <= len - 3) fail = !tap5_fast(w[k], w[k + 1], w[k + 2], w[k + 3], w[k + 4], &r);
                        if (!fail) {
                            P.out[v] = r;
                            if (STATS) acc.add(r, gx, gy, pos, P.iso);
                        }
                    }
                    F.push(fail, v, lane);
                }
            }
            F.drain(P, acc, lane);
        }
    }
    F.finish(P, acc, lane);
    if (STATS) acc.flush(P.st, true);
}

// resident CTAs of a kernel on the current device, or 0 when the query fails
int resident_blocks(const void *fn, int threads) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return sms * std::max(per_sm, 1);
}

constexpr int KRUN = 8, KSEG = 8;

// resident CTAs of each pass kernel, per device ordinal: queried on the first
// call on that device and kept once every query succeeded (a failed query
// gives 4 CTAs per SM of this call's device and is asked again next time)
struct PassGrids {
    int x, x4, a, z;
};
PassGrids pass_grids() {
    static std::mutex mu;
    static std::map<int, PassGrids> known;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) cudaGetLastError();
    {
        std::lock_guard<std::mutex> lk(mu);
        auto it = known.find(dev);
        if (it != known.end()) return it->second;
    }
    PassGrids g{resident_blocks((const void *)k_pass_x, 256), resident_blocks((const void *)k_pass_x4, 256),
                resident_blocks((const void *)k_pass_axis<KRUN, KSEG, false>, 256),
                resident_blocks((const void *)k_pass_axis<KRUN, KSEG, true>, 256)};
    if (g.x && g.x4 && g.a && g.z) {
        std::lock_guard<std::mutex> lk(mu);
        known[dev] = g;
        return g;
    }
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) {
        cudaGetLastError();
        sms = 152;
    }
    if (!g.x) g.x = 4 * sms;
    if (!g.x4) g.x4 = 4 * sms;
    if (!g.a) g.a = 4 * sms;
    if (!g.z) g.z = 4 * sms;
    return g;
}
}  // namespace

bool smooth_can_stage(int nx, int ny, int nz) { return (size_t)nx * ny * nz < ((size_t)1 << 32); }

// three passes; row and slice indices are 32-bit, so volumes stay below 2^32
// voxels (meshify accepts at most 2^31-1)
n2m_status launch_smooth(const float *in, float *out, float *tmp, int nx, int ny, int nz, float iso, VolStats *st,
                         cudaStream_t s, const StagedInput *stage) {
    const size_t n = (size_t)nx * ny * nz;
    if (n >= ((size_t)1 << 32)) {
        n2m_set_error("smoothing supports fewer than 2^32 voxels");
        return N2M_ERR_TOO_LARGE;
    }
    const PassGrids G = pass_grids();
    const int gx = G.x, gx4 = G.x4, ga = G.a, gz = G.z;
    const unsigned nxy = (unsigned)nx * ny;
    const Pass px{in, out, 1u, nx, ny, nxy, iso, st}, py{out, tmp, (unsigned)nx, nx, ny, nxy, iso, st},
        pz{tmp, out, nxy, nx, ny, nxy, iso, st};
    // 16-byte rows: the float4 x pass
    const bool x4 = nx % 4 == 0 && ((uintptr_t)in & 15) == 0 && ((uintptr_t)out & 15) == 0;
    auto pass_x = [&](unsigned r0, unsigned r1, unsigned g) -> n2m_status {
        if (x4) n2m_launch(k_pass_x4, std::min<unsigned>(g, (unsigned)gx4), 256, 0, s, px, r0, r1);
        else n2m_launch(k_pass_x, std::min<unsigned>(g, (unsigned)gx), 256, 0, s, px, r0, r1);
        CKL();
        return N2M_OK;
    };
    if (stage && stage->host) {
        // the copy stream may only overwrite `in` once earlier work on s is done with it
        CK(cudaEventRecord(stage->ev[N2M_STAGE_SLABS], s));
        CK(cudaStreamWaitEvent(stage->copy, stage->ev[N2M_STAGE_SLABS], 0));
        // per slab: x and y passes as soon as it has arrived, then the z pass of
        // every slice whose five y-pass inputs are done
        int zdone = 0;
        for (int k = 0; k < N2M_STAGE_SLABS; k++) {
            const int z0 = (int)((long long)nz * k / N2M_STAGE_SLABS), z1 = (int)((long long)nz * (k + 1) / N2M_STAGE_SLABS);
            if (z1 <= z0) continue;
            const size_t off = (size_t)z0 * nxy, bytes = (size_t)(z1 - z0) * nxy * sizeof(float);
            CK(cudaMemcpyAsync((float *)in + off, stage->host + off, bytes, cudaMemcpyHostToDevice, stage->copy));
            CK(cudaEventRecord(stage->ev[k], stage->copy));
            CK(cudaStreamWaitEvent(s, stage->ev[k], 0));
            const unsigned r0 = (unsigned)z0 * ny, r1 = (unsigned)z1 * ny;
            CKS(pass_x(r0, r1, std::max<unsigned>(1u, (r1 - r0 + 7) / 8)));
            n2m_launch(k_pass_axis<KRUN, KSEG, false>, ga, 256, 0, s, py, ny, (unsigned)z0, (unsigned)(z1 - z0), 0,
                       ny);
            const int zready = z1 == nz ? nz : z1 - 2;
            if (zready > zdone) {
                n2m_launch(k_pass_axis<KRUN, KSEG, true>, gz, 256, 0, s, pz, nz, 0u, 1u, zdone, zready);
                zdone = zready;
            }
        }
    } else {
        CKS(pass_x(0u, (unsigned)ny * nz, 0xffffffffu));
        n2m_launch(k_pass_axis<KRUN, KSEG, false>, ga, 256, 0, s, py, ny, 0u, (unsigned)nz, 0, ny);
        n2m_launch(k_pass_axis<KRUN, KSEG, true>, gz, 256, 0, s, pz, nz, 0u, 1u, 0, nz);
    }
    CKL();
    return N2M_OK;
}

namespace {
// transposed 5-tap pass along one axis: out_j = sum over interior rows i with
// |i-j| <= 2 of w_|i-j| g_i, plus g_j where j itself is a row left unfiltered
__global__ void k_smooth_T(const float *__restrict__ g, float *__restrict__ out, int nx, int ny, int nz, int axis) {
    grid_wait();
    const long long n = (long long)nx * ny * nz;
    const long long stride = axis == 0 ? 1 : (axis == 1 ? nx : (long long)nx * ny);
    const int len = axis == 0 ? nx : (axis == 1 ? ny : nz);
    const float w[3] = {0.45f, 0.225f, 0.05f};
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        const long long q = v / stride;
        const int j = (int)(axis == 0 ? q % nx : (axis == 1 ? q % ny : q));
        float acc = (j < 2 || j > len - 3) ? g[v] : 0.f;
        for (int d = -2; d <= 2; d++) {
            const int i = j + d;
            if (i >= 2 && i <= len - 3) acc += w[d < 0 ? -d : d] * g[v + d * stride];
        }
        out[v] = acc;
    }
}
}  // namespace

n2m_status launch_smooth_adjoint(const float *g, float *tmp, float *out, int nx, int ny, int nz, cudaStream_t s) {
    const long long n = (long long)nx * ny * nz;
    const unsigned blocks = (unsigned)std::min<long long>((n + 255) / 256, 152 * 64);
    n2m_launch(k_smooth_T, blocks, 256, 0, s, g, out, nx, ny, nz, 2);
    n2m_launch(k_smooth_T, blocks, 256, 0, s, out, tmp, nx, ny, nz, 1);
    n2m_launch(k_smooth_T, blocks, 256, 0, s, tmp, out, nx, ny, nz, 0);
    CKL();
    return N2M_OK;
}

n2m_status launch_stats(const float *vol, int nx, int ny, int nz, float iso, bool minmax, VolStats *st,
                        cudaStream_t s, int z0) {
    const long long rows = (long long)ny * nz;
    const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>((rows + 7) / 8, 152 * 8));   // 8 rows per block
    n2m_launch(k_stats, grid, 256, 0, s, vol, nx, ny, nz, z0, iso, st, minmax);
    CKL();
    return N2M_OK;
}

// ==== pre-smooth with exact rounding on demand ===================================
// Marching cubes reads the smoothed volume in two ways only: the sign of every
// grid point (value >= iso, and value - iso against the FLT_EPSILON clamp), and
// the values at the ends of the edges the surface crosses and at the corners of
// ambiguous cubes.  So the volume
// is first smoothed approximately in one fused FP32 pass (pass A: one read and
// one write per voxel), with a rigorous error bound; the few voxels whose sign
// the bound leaves open, and the candidates for the volume's minimum and
// maximum, are recomputed with the reference's double sequence (pass B).
// With the sign words the voxels whose values will be read are marked
// (mcwords.cuh: k_words) and the exact three-pass smoothing runs on those voxels
// only, the x and y passes on the voxels those depend on (marks dilated by +-2
// slices, then +-2 rows), by lists of bit words.  Every value
// marching cubes reads is then the reference's float, bit for bit.
//
// Error bound of pass A: each pass evaluates the tap sum as an FP32 FMA chain
// with the weights rounded to float: at most 7 * 2^-24 * M from the reference's
// float of the same inputs (M = the largest input magnitude in the window; the
// weights sum to 1, so every partial sum is below M), and the errors of earlier
// passes carry through with total weight 1: after three passes at most
// 21 * 2^-24 * M < 2^-19 * M, M being any bound on the input magnitudes the
// voxel depends on.  A warp uses the largest magnitude it has read so far.
namespace {
constexpr float OW0 = 0.45f, OW1 = 0.225f, OW2 = 0.05f;

// two floats in one 64-bit register pair: each instruction works on both halves, rounded as the scalar one rounds
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// three-input minimum and maximum (a NaN operand is ignored, as by fminf and fmaxf)
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ f2 tap2(f2 a, f2 b, f2 c, f2 d, f2 e, f2 w0, f2 w1, f2 w2) {
    return fma2(e, w2, fma2(d, w1, fma2(c, w0, fma2(b, w1, mul2(a, w2)))));
}
__device__ __forceinline__ float fma5(float a, float b, float c, float d, float e) {
    return __fmaf_rn(e, OW2, __fmaf_rn(d, OW1, __fmaf_rn(c, OW0, __fmaf_rn(b, OW1, __fmul_rn(a, OW2)))));
}

__device__ __forceinline__ void od_flag(OdStats *st, unsigned f) { atomicOr(&st->flags, f); }

// ---- TMA and mbarrier primitives (inline PTX) ----
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, unsigned long long *bar, int x, int y,
                                            int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}
// order this thread's earlier generic-proxy accesses to shared memory before later TMA writes
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Pass A: the input volume through a TMA tensor map, whose rows begin at multiples of 16
// bytes.  ODD: nx is no multiple of 4 or the volume itself is not aligned; the map
// then is of a copy with padded rows (k_od_pad), and the output, whose rows begin
// anywhere, is written value by value.  The exact three passes, the other way to smooth such a
// volume, read and write every voxel three times: 511 x 512 x 512 CT 2241 us, 1630 this way,
// clustered 2514 and 1670, 333^3 870 and 740, 2 to 7 M voxels within 4 %.  Boxes of 72 x 12 x 1 floats, x0 - 4 ..
// x0 + 67 and y0 - 2 .. y0 + 9 of one slice (outside the volume the copy fills
// zeros).  A warp takes 64 x 8 columns of `zrun` slices; its lane 0 keeps OA_S
// slices in flight in the warp's own ring of shared-memory stages, each
// completing on its mbarrier.  A lane owns 4 consecutive columns (one 16-byte
// load per row, two register pairs) of 4 rows, lanes 0-15 the tile's upper rows
// and 16-31 its lower ones.  The passes run y, z, x: the y pass over the 8 loaded
// rows and the z pass over a five-slice register ring stay inside a lane and use
// the paired FP32 instructions; only the x pass needs neighbours, two values from
// each side per row, by shuffle.  The two columns beyond either end of a tile row
// are 16 (column, row) pairs, one per lane, that take the same y and z passes.
// The separable filter's axes commute, so the order does not enter the bound.
// Each output is classified on the spot: |v - iso| <= B + 4 eps -> listed as
// undecided, else its sign goes to the bitmap and, when positive, the bbox.  A
// task leaves its minimum, maximum and B for k_od_scan and offers min + B
// (max - B) as a bound on the volume's exact extreme.  Waits give up after a fixed
// number of polls (flag OD_TIMEOUT), after waiting, also bounded, for the warp's
// copies still in flight.
//
// 512^3: 1.09 GB (8.15 bytes a voxel) in 255 us = 4.3 TB/s, 38 instructions a voxel at
// 53 % of the issue slots: the register ring allows 12 warps per SM, and their
// dependent FP32 chains and the half-rate min/max and shifts bound it.  With one column
// and 8 rows per lane (x pass first, five shared-memory loads per row, 92
// instructions a voxel) it took 479 us.  Two rows per lane (more warps, twice the halo
// rows): 292 us; a fourth CTA per SM (spills): 423 us.
constexpr int OA_R = 4, OA_S = 4, OA_X = 64, OA_Y = 2 * OA_R, OA_BW = OA_X + 8, OA_BH = OA_Y + 4, OA_WARPS = 4;
constexpr unsigned OA_BYTES = OA_BW * OA_BH * 4;
constexpr int OA_POLLS = 1 << 22;
struct __align__(128) OaStage {
    float v[OA_BH][OA_BW];
};

// OR over the eight lanes that share a 32-voxel word, of the lane's four rows' words at once: lane i of the eight
// ends up with the word of row word_row(i)
__device__ __forceinline__ int word_row(int lane) { return (lane & 1) * 2 + (lane >> 1 & 1); }
__device__ __forceinline__ unsigned or_rows(const unsigned (&p)[OA_R], int lane) {
    const unsigned FULL = 0xffffffffu;
    const bool b0 = lane & 1, b1 = lane & 2;
    unsigned k0 = b0 ? p[2] : p[0], k1 = b0 ? p[3] : p[1];
    k0 |= __shfl_xor_sync(FULL, b0 ? p[0] : p[2], 1);
    k1 |= __shfl_xor_sync(FULL, b0 ? p[1] : p[3], 1);
    unsigned k = b1 ? k1 : k0;
    k |= __shfl_xor_sync(FULL, b1 ? k0 : k1, 2);
    return k | __shfl_xor_sync(FULL, k, 4);
}

// lists the lane's undecided voxels (any: it has some), in `rows` rows of `cols` from p; returns its row word's bits of them.
// Out of line: rare, and the kernel's slice loop is unrolled five times.  With the isolevel on a plateau (a mask meshed at
// its own value) half the volume comes here: one atomic per warp, and none once the list is full and the caller falls
// back anyway (1.4 M voxels of a 181 x 217 x 181 mask, an atomic each: 0.83 ms for the exact smoothing with the attempt).
__device__ __noinline__ unsigned list_undecided(const float *p, int nx, int rows, int cols, unsigned j, bool any, float band, float iso,
                                                unsigned *cnt, unsigned *list, unsigned cap, int lane) {
    const unsigned FULL = 0xffffffffu;
    const unsigned listed = lane == 0 ? *(volatile unsigned *)cnt : 0u;
    if (__shfl_sync(FULL, listed, 0) > cap) return 0u;
    unsigned uw[OA_R], mine = 0u;
#pragma unroll
    for (int r = 0; r < OA_R; r++) {
        unsigned m = 0u;
        for (int c = 0; any && r < rows && c < cols; c++)
            if (fabsf(__fsub_rn(p[(size_t)r * nx + c], iso)) <= band) m |= 1u << (4 * (lane & 7) + c);
        uw[r] = m;
        mine += __popc(m);
    }
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    unsigned at = lane == 31 ? atomicAdd(cnt, incl) : 0u;
    at = __shfl_sync(FULL, at, 31) + incl - mine;
#pragma unroll
    for (int r = 0; r < OA_R; r++)
        for (unsigned m = uw[r]; m; m &= m - 1u, at++)
            if (at < cap) list[at] = j + (unsigned)(r * nx + (__ffs(m) - 1 - 4 * (lane & 7)));
    return or_rows(uw, lane);
}

template <bool ODD>
__global__ void __launch_bounds__(OA_WARPS * 32, 3) k_od_approx(const __grid_constant__ CUtensorMap tmap, float *out,
                                                             int nx, int ny, int nz, int zrun, float iso, OdStats *st,
                                                             OdLists L) {
    grid_wait();
    const unsigned FULL = 0xffffffffu;
    __shared__ OaStage stage[OA_WARPS][OA_S];
    __shared__ unsigned long long bars[OA_WARPS][OA_S];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, seg = lane >> 4, li = lane & 15;
    OaStage *sg = stage[wid];
    unsigned long long *bw = bars[wid];
    if (lane == 0) {
        for (int k = 0; k < OA_S; k++) mbar_init(&bw[k], 1);
        mbar_fence_init();
    }
    __syncwarp();
    unsigned issued = 0, used = 0;   // loads issued / consumed by this warp (stage = n % OA_S, parity = n / OA_S)
    const unsigned nxs = (unsigned)(nx + OA_X - 1) / OA_X, nys = (unsigned)(ny + OA_Y - 1) / OA_Y;
    const unsigned ntask = nxs * nys * ((unsigned)(nz + zrun - 1) / (unsigned)zrun);
    const size_t nxy = (size_t)nx * ny;
    const f2 w0 = pack2(OW0, OW0), w1 = pack2(OW1, OW1), w2 = pack2(OW2, OW2), zero2 = pack2(0.f, 0.f), niso2 = pack2(-iso, -iso);
    // this lane's halo column and row: columns x0-2, x0-1, x0+64, x0+65
    const int hc = (li / OA_R) & 3, hr = li % OA_R, hcol = hc < 2 ? 2 + hc : OA_X + 2 + hc;
    bool timed_out = false;
    for (unsigned task = blockIdx.x * OA_WARPS + wid; task < ntask && !timed_out; task += gridDim.x * OA_WARPS) {
        const unsigned xs = task % nxs, t2 = task / nxs;
        const int x0 = (int)xs * OA_X, y0 = (int)(t2 % nys) * OA_Y, zs = (int)(t2 / nys) * zrun, ze = min(zs + zrun, nz);
        const int x = x0 + 4 * li, y = y0 + OA_R * seg;   // first column and row of this lane
        const bool ownx = x < nx;
        const int cols = ODD ? min(4, nx - x) : 4;   // columns of this lane inside the volume
        const bool xedge = x0 == 0 || x0 + OA_X >= nx - 1, yedge = y0 < 2 || y0 + OA_Y > ny - 2;
        // every slice zs-2 .. ze+1 is loaded (outside the volume: zeros, read only by outputs that ignore them)
        int znext = zs - 2;
        const int zlast = ze + 1;
        auto issue = [&]() {
            if (lane == 0) {
                const unsigned k = issued % OA_S;
                fence_proxy_async();
                mbar_expect_tx(&bw[k], OA_BYTES);
                tma_load_3d(&sg[k], &tmap, &bw[k], x0 - 4, y0 - 2, znext);
            }
            issued++;
            znext++;
        };
        while (znext <= zlast && issued - used < (unsigned)OA_S) issue();
        f2 zr[5][OA_R][2];   // y values of five slices
        float hz[5];
#pragma unroll
        for (int a = 0; a < 5; a++) {
            hz[a] = 0.f;
#pragma unroll
            for (int r = 0; r < OA_R; r++) zr[a][r][0] = zr[a][r][1] = zero2;
        }
        float mrun = 0.f, lmin = INFINITY, lmax = -INFINITY, B = 0.f;
        int bzl = INT_MAX, bzh = INT_MIN;
        unsigned orx = 0;      // this lane's row word, over the slices: columns with a decided voxel >= iso
        f2 nanacc = zero2;     // becomes NaN if an output is NaN or infinite
        for (int zb = zs - 2; zb <= zlast && !timed_out; zb += 5) {
#pragma unroll
            for (int u = 0; u < 5; u++) {   // ring slot u takes slice zb + u
                const int zi = zb + u;
                if (zi > zlast) break;
                const unsigned k = used % OA_S, par = (used / OA_S) & 1u;
                bool ok = false;
                for (int it = 0; it < OA_POLLS && !ok; it++) ok = mbar_try_wait(&bw[k], par);
                if (!__all_sync(FULL, ok)) {
                    timed_out = true;
                    break;
                }
                const OaStage &S = sg[k];
                f2 in[OA_R + 4][2];
#pragma unroll
                for (int r = 0; r < OA_R + 4; r++) {
                    const ulonglong2 q = *(const ulonglong2 *)&S.v[OA_R * seg + r][4 + 4 * li];
                    in[r][0] = q.x;
                    in[r][1] = q.y;
                    float a, b, c, d;
                    unpack2(q.x, a, b);
                    unpack2(q.y, c, d);
                    mrun = max3(max3(mrun, fabsf(a), fabsf(b)), fabsf(c), fabsf(d));
                }
                float hv;
                {
                    const float *q = &S.v[OA_R * seg + hr][hcol];
                    const float a = q[0], b = q[OA_BW], c = q[2 * OA_BW], d = q[3 * OA_BW], e = q[4 * OA_BW];
                    mrun = fmaxf(max3(max3(mrun, fabsf(a), fabsf(b)), fabsf(c), fabsf(d)), fabsf(e));
                    hv = fma5(a, b, c, d, e);
                    if (yedge && (y + hr < 2 || y + hr > ny - 3)) hv = c;
                }
#pragma unroll
                for (int r = 0; r < OA_R; r++)
#pragma unroll
                    for (int h = 0; h < 2; h++)
                        zr[u][r][h] = tap2(in[r][h], in[r + 1][h], in[r + 2][h], in[r + 3][h], in[r + 4][h], w0, w1, w2);
                if (yedge) {
#pragma unroll
                    for (int r = 0; r < OA_R; r++)
                        if (y + r < 2 || y + r > ny - 3) {
                            zr[u][r][0] = in[r + 2][0];
                            zr[u][r][1] = in[r + 2][1];
                        }
                }
                hz[u] = hv;
                __syncwarp();   // every lane is done with the stage
                used++;
                if (znext <= zlast) issue();
                // bounds every output whose inputs have been read
                B = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(mrun))) * 0x1p-19f;
                const int z = zi - 2;
                if (z < zs) continue;
                constexpr int P = 5;
                const int s0 = (u + 1) % P, s1 = (u + 2) % P, s2 = (u + 3) % P, s3 = (u + 4) % P;   // slices z-2 .. z+1
                const bool zint = z >= 2 && z <= nz - 3;
                const float hy = zint ? fma5(hz[s0], hz[s1], hz[s2], hz[s3], hz[u]) : hz[s2];
                const float band = B + 4.0f * N2M_FLT_EPS;
                float *op = out + (size_t)z * nxy + (size_t)y * nx + x;
                unsigned pw[OA_R];
                float dmin = INFINITY;
#pragma unroll
                for (int r = 0; r < OA_R; r++) {
                    f2 va = zr[s2][r][0], vb = zr[s2][r][1];
                    if (zint) {
                        va = tap2(zr[s0][r][0], zr[s1][r][0], va, zr[s3][r][0], zr[u][r][0], w0, w1, w2);
                        vb = tap2(zr[s0][r][1], zr[s1][r][1], vb, zr[s3][r][1], zr[u][r][1], w0, w1, w2);
                    }
                    float v0, v1, v2, v3;
                    unpack2(va, v0, v1);
                    unpack2(vb, v2, v3);
                    const float h1 = __shfl_sync(FULL, hy, li == 0 ? r : 2 * OA_R + r, 16), h2 = __shfl_sync(FULL, hy, li == 0 ? OA_R + r : 3 * OA_R + r, 16);
                    float l2 = __shfl_up_sync(FULL, v2, 1, 16), l3 = __shfl_up_sync(FULL, v3, 1, 16);
                    float r0 = __shfl_down_sync(FULL, v0, 1, 16), r1 = __shfl_down_sync(FULL, v1, 1, 16);
                    l2 = li == 0 ? h1 : l2;
                    l3 = li == 0 ? h2 : l3;
                    r0 = li == 15 ? h1 : r0;
                    r1 = li == 15 ? h2 : r1;
                    const f2 m1 = pack2(v1, v2);
                    f2 oa = tap2(pack2(l2, l3), pack2(l3, v0), va, m1, vb, w0, w1, w2);
                    f2 ob = tap2(va, m1, vb, pack2(v3, r0), pack2(r0, r1), w0, w1, w2);
                    if (xedge) {   // columns 0, 1 and nx-2, nx-1 keep their value
                        if (x == 0) oa = va;
                        if (!ODD && x + 4 == nx) ob = vb;
                        if (ODD && x + 6 > nx) {   // columns past the volume repeat the lane's first
                            float o0, o1, o2, o3;
                            unpack2(oa, o0, o1);
                            unpack2(ob, o2, o3);
                            if (x + 2 >= nx) o0 = v0;
                            if (x + 3 >= nx) o1 = cols > 1 ? v1 : o0;
                            if (x + 4 >= nx) o2 = cols > 2 ? v2 : o0;
                            if (x + 5 >= nx) o3 = cols > 3 ? v3 : o0;
                            oa = pack2(o0, o1);
                            ob = pack2(o2, o3);
                        }
                    }
                    pw[r] = 0u;
                    if (ownx && y + r < ny) {
                        if (ODD) {   // rows begin anywhere
                            float *q = op + (size_t)r * nx, o0, o1, o2, o3;
                            unpack2(oa, o0, o1);
                            unpack2(ob, o2, o3);
                            q[0] = o0;
                            if (cols > 1) q[1] = o1;
                            if (cols > 2) q[2] = o2;
                            if (cols > 3) q[3] = o3;
                        } else {
                            *(ulonglong2 *)(op + (size_t)r * nx) = make_ulonglong2(oa, ob);
                        }
                        nanacc = fma2(oa, zero2, fma2(ob, zero2, nanacc));
                        float o0, o1, o2, o3;
                        unpack2(oa, o0, o1);
                        unpack2(ob, o2, o3);
                        lmin = min3(min3(lmin, o0, o1), o2, o3);
                        lmax = max3(max3(lmax, o0, o1), o2, o3);
                        unpack2(add2(oa, niso2), o0, o1);
                        unpack2(add2(ob, niso2), o2, o3);
                        dmin = min3(min3(dmin, fabsf(o0), fabsf(o1)), fabsf(o2), fabsf(o3));
                        // sign bits (the exact sign of every decided voxel; pass B sets the others)
                        unsigned n = __float_as_uint(o3) >> 31;
                        n = __funnelshift_l(__float_as_uint(o2), n, 1);
                        n = __funnelshift_l(__float_as_uint(o1), n, 1);
                        n = __funnelshift_l(__float_as_uint(o0), n, 1);
                        pw[r] = ((n ^ 15u) & (ODD ? (1u << cols) - 1u : 15u)) << (4 * (li & 7));
                    }
                }
                const unsigned word = or_rows(pw, lane);
                unsigned dec = word;
                if (__any_sync(FULL, dmin <= band)) {   // list the undecided voxels (their values are in `out`)
                    dec &= ~list_undecided(op, nx, min(OA_R, ny - y), cols, (unsigned)((size_t)z * nxy + (size_t)y * nx + x), dmin <= band,
                                           band, iso, L.cnt, L.unc, L.cap, lane);
                }
                const int row = word_row(lane);
                if (!(lane & 4) && x0 + (li & 8) * 4 < nx)
                    L.vsign[od_vsign_word((unsigned)(x0 + (li & 8) * 4), (unsigned)(y + row), (unsigned)z, L.wv, L.nys)] = word;
                if (dec) {
                    orx |= dec;
                    bzl = min(bzl, z);
                    bzh = z;
                }
            }
        }
        if (timed_out) break;
        const bool full = *(volatile unsigned *)L.cnt > L.cap;   // of undecided voxels: the caller falls back
        // huge, infinite or NaN input (an unbounded B), or a non-finite output
        float na, nb;
        unpack2(nanacc, na, nb);
        const bool bad = !(B < 0x1p+120f * 0x1p-19f) || na != 0.f || nb != 0.f;
        if (__any_sync(FULL, bad)) {   // the exact three-pass path handles the volume
            if (lane == 0) od_flag(st, OD_FALLBACK);
            continue;
        }
        // bbox of the decided voxels >= iso; an atomic only where it may still change something
        if (__any_sync(FULL, orx != 0u)) {
            const int gx = x0 + (li & 8) * 4, row = y + word_row(lane);
            const int xl = __reduce_min_sync(FULL, orx ? gx + __ffs(orx) - 1 : INT_MAX);
            const int xh = __reduce_max_sync(FULL, orx ? gx + 31 - __clz(orx) : INT_MIN);
            const int yl = __reduce_min_sync(FULL, orx ? row : INT_MAX), yh = __reduce_max_sync(FULL, orx ? row : INT_MIN);
            const int zl = __reduce_min_sync(FULL, bzl), zh = __reduce_max_sync(FULL, bzh);
            if (lane < 3) {
                const int lo = lane == 0 ? xl : (lane == 1 ? yl : zl), hi = lane == 0 ? xh : (lane == 1 ? yh : zh);
                if (lo < *(volatile int *)&st->vs.lo[lane]) atomicMin(&st->vs.lo[lane], lo);
                if (hi > *(volatile int *)&st->vs.hi[lane]) atomicMax(&st->vs.hi[lane], hi);
            }
        }
        for (int o = 16; o; o >>= 1) {
            lmin = fminf(lmin, __shfl_xor_sync(FULL, lmin, o));
            lmax = fmaxf(lmax, __shfl_xor_sync(FULL, lmax, o));
        }
        if (lane == 0) {
            L.range[task] = make_float4(lmin, lmax, B, 0.f);
            const int um = f2ord(__fadd_ru(lmin, B)), lm = f2ord(__fsub_rd(lmax, B));
            if (um < *(volatile int *)&st->umin) atomicMin(&st->umin, um);
            if (lm > *(volatile int *)&st->lmax) atomicMax(&st->lmax, lm);
        }
        if (__any_sync(FULL, full)) break;
    }
    if (timed_out) {
        // no further copies are issued; wait (bounded) for the ones in flight before leaving
        if (lane == 0) od_flag(st, OD_FALLBACK | OD_TIMEOUT);
        while (used < issued) {
            const unsigned k = used % OA_S, par = (used / OA_S) & 1u;
            for (int it = 0; it < OA_POLLS; it++)
                if (mbar_try_wait(&bw[k], par)) break;
            used++;
        }
    }
}

// The voxels that can still be the volume's extreme: those of a task whose minimum
// (maximum) can, with a value within B of the bound.  A block looks at OS_T tasks and
// reads the few that qualify again with all its warps, a slice's 16 loads of a warp in
// flight at once (a warp per task and one row after another took 246 us for the
// 512^3 CT volume's handful).  A list that is full (a plateau at that extreme) takes no
// more; k_od_resolve then finds that extreme without it.  8.4 us for the 512^3 CT volume; 73
// padded with one value (107 with an atomic per voxel there too).
constexpr int OS_T = 64;
constexpr unsigned OD_SAMPLE = 4096;   // at most a list's capacity
__global__ void __launch_bounds__(256) k_od_scan(const float *__restrict__ out, int nx, int ny, int nz, int zrun,
                                                 OdStats *st, OdLists L) {
    grid_wait();
    __shared__ unsigned todo[OS_T], ntodo;
    const unsigned flags = st->flags, undecided = st->cnt[0];   // read together
    if (flags || undecided > L.cap) return;   // not every task has a range
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned nxs = (unsigned)(nx + OA_X - 1) / OA_X, nys = (unsigned)(ny + OA_Y - 1) / OA_Y;
    const unsigned ntask = nxs * nys * ((unsigned)(nz + zrun - 1) / (unsigned)zrun);
    const float umin = ord2f(st->umin), lmax = ord2f(st->lmax);
    const size_t nxy = (size_t)nx * ny;
    if (threadIdx.x == 0) ntodo = 0u;
    __syncthreads();
    if (threadIdx.x < OS_T) {
        const unsigned task = blockIdx.x * OS_T + threadIdx.x;
        const float4 t = task < ntask ? L.range[task] : make_float4(0.f, 0.f, 0.f, 0.f);
        if (task < ntask && (__fsub_rd(t.x, t.z) <= umin || __fadd_ru(t.y, t.z) >= lmax)) todo[atomicAdd(&ntodo, 1u)] = task;
    }
    __syncthreads();
    // bit k of m: the lane's voxel of row k / 2, columns 32 (k & 1) on, j being that of k = 0; one atomic per warp
    auto put = [&](unsigned m, unsigned j, unsigned *n, unsigned *list) {
        if (!__any_sync(FULL, m != 0u)) return;
        unsigned incl = __popc(m);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        unsigned at = lane == 31 ? atomicAdd(n, incl) : 0u;
        at = __shfl_sync(FULL, at, 31) + incl - __popc(m);
        for (; m; m &= m - 1u, at++) {
            const unsigned k = (unsigned)__ffs(m) - 1u;
            if (at < L.cap) list[at] = j + (k >> 1) * (unsigned)nx + 32u * (k & 1u);
        }
    };
    unsigned open = 3u;   // lists (1: minimum, 2: maximum) that this warp has not seen full
    for (unsigned i = 0; i < ntodo; i++) {
        const unsigned task = todo[i], xs = task % nxs, t2 = task / nxs;
        const float4 t = L.range[task];
        const unsigned want = (__fsub_rd(t.x, t.z) <= umin ? 1u : 0u) | (__fadd_ru(t.y, t.z) >= lmax ? 2u : 0u);
        if (!(want & open)) continue;
        if (i) {   // (the first task, often the only one, waits for no count)
            const unsigned room = (*(volatile unsigned *)&L.cnt[1] <= L.cap ? 1u : 0u) | (*(volatile unsigned *)&L.cnt[2] <= L.cap ? 2u : 0u);
            open &= __shfl_sync(FULL, room, 0);
        }
        const bool mn = want & open & 1u, mx = want & open & 2u;   // the same for the whole warp
        if (!mn && !mx) continue;
        const int x0 = (int)xs * OA_X, y0 = (int)(t2 % nys) * OA_Y, zs = (int)(t2 / nys) * zrun, ze = min(zs + zrun, nz);
        for (int z = zs + wid; z < ze; z += 8) {
            float v[2 * OA_Y];
#pragma unroll
            for (int k = 0; k < 2 * OA_Y; k++) {
                const int x = x0 + 32 * (k & 1) + lane, y = y0 + (k >> 1);
                v[k] = x < nx && y < ny ? out[(size_t)z * nxy + (size_t)y * nx + x] : NAN;
            }
            const unsigned j0 = (unsigned)((size_t)z * nxy + (size_t)y0 * nx + x0 + lane);
            // a plateau shows in the middle row (votes for every row would cost the usual few candidates 1 us)
            if (mn && __all_sync(FULL, !(__fsub_rd(v[OA_Y], t.z) > umin))) {
                unsigned m = 0u;
#pragma unroll
                for (int k = 0; k < 2 * OA_Y; k++) m |= (__fsub_rd(v[k], t.z) <= umin ? 1u : 0u) << k;
                put(m, j0, &L.cnt[1], L.cmin);
            } else if (mn) {
#pragma unroll
                for (int k = 0; k < 2 * OA_Y; k++)   // a NaN is in neither list
                    if (__fsub_rd(v[k], t.z) <= umin) {
                        const unsigned q = atomicAdd(&L.cnt[1], 1u);
                        if (q < L.cap) L.cmin[q] = j0 + (unsigned)((k >> 1) * nx + 32 * (k & 1));
                    }
            }
            if (mx && __all_sync(FULL, !(__fadd_ru(v[OA_Y], t.z) < lmax))) {
                unsigned m = 0u;
#pragma unroll
                for (int k = 0; k < 2 * OA_Y; k++) m |= (__fadd_ru(v[k], t.z) >= lmax ? 1u : 0u) << k;
                put(m, j0, &L.cnt[2], L.cmax);
            } else if (mx) {
#pragma unroll
                for (int k = 0; k < 2 * OA_Y; k++)
                    if (__fadd_ru(v[k], t.z) >= lmax) {
                        const unsigned q = atomicAdd(&L.cnt[2], 1u);
                        if (q < L.cap) L.cmax[q] = j0 + (unsigned)((k >> 1) * nx + 32 * (k & 1));
                    }
            }
        }
    }
}

// Plateaus.  Every step of a tap (products with positive weights, sums, roundings) is monotone in
// each input, so a voxel filtered along k axes is nowhere below tap^k(m), m the smallest raw value
// it depends on, nor above tap^k(M).  Its other axes leave it in their face layers (0, 1, n - 2,
// n - 1), and everything it depends on in the same ones, so m and M are the extremes of the raw
// voxels in the face layers of at least 3 - k axes: r[c], c = 3 - k.
__device__ __forceinline__ void raw_extremes(const float *__restrict__ in, int nx, int ny, int nz, OdStats *st) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    float lo[4], hi[4];   // of the voxels in the face layers of at least c axes
#pragma unroll
    for (int c = 0; c < 4; c++) {
        lo[c] = INFINITY;
        hi[c] = -INFINITY;
    }
    const unsigned nrows = (unsigned)ny * (unsigned)nz;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrows; r += (gridDim.x * blockDim.x) >> 5) {
        const int z = (int)(r / (unsigned)ny), y = (int)(r - (unsigned)z * (unsigned)ny);
        const int faces = (y < 2 || y > ny - 3) + (z < 2 || z > nz - 3);
        const float *p = in + (size_t)r * nx;
        float il = INFINITY, ih = -INFINITY, el = INFINITY, eh = -INFINITY;   // away from the x faces, in them
#pragma unroll 8
        for (int x = lane; x < nx; x += 32) {
            const float v = __ldg(p + x);
            if (x < 2 || x > nx - 3) {
                el = fminf(el, v);
                eh = fmaxf(eh, v);
            } else {
                il = fminf(il, v);
                ih = fmaxf(ih, v);
            }
        }
#pragma unroll
        for (int c = 0; c < 4; c++) {
            if (faces >= c) {
                lo[c] = fminf(lo[c], il);
                hi[c] = fmaxf(hi[c], ih);
            }
            if (faces + 1 >= c) {
                lo[c] = fminf(lo[c], el);
                hi[c] = fmaxf(hi[c], eh);
            }
        }
    }
    __shared__ int bl[4], bh[4];
    if (threadIdx.x < 4) {
        bl[threadIdx.x] = INT_MAX;
        bh[threadIdx.x] = INT_MIN;
    }
    __syncthreads();
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const int l = __reduce_min_sync(FULL, f2ord(lo[c])), h = __reduce_max_sync(FULL, f2ord(hi[c]));
        if (lane == 0) {
            atomicMin(&bl[c], l);
            atomicMax(&bh[c], h);
        }
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        if (bl[threadIdx.x] < *(volatile int *)&st->rlo[threadIdx.x]) atomicMin(&st->rlo[threadIdx.x], bl[threadIdx.x]);
        if (bh[threadIdx.x] > *(volatile int *)&st->rhi[threadIdx.x]) atomicMax(&st->rhi[threadIdx.x], bh[threadIdx.x]);
    }
}
// whether the extremes found among some of the candidates are the bounds above, which makes them the volume's
__device__ __forceinline__ bool plateau_holds(const OdStats *st, bool low, bool high) {
    float mn = INFINITY, mx = -INFINITY;
    for (int c = 0; c < 4; c++) {
        float l = ord2f(*(volatile const int *)&st->rlo[c]), h = ord2f(*(volatile const int *)&st->rhi[c]);
        for (int k = c; k < 3; k++) {
            l = tap5_double(l, l, l, l, l);
            h = tap5_double(h, h, h, h, h);
        }
        mn = fminf(mn, l);
        mx = fmaxf(mx, h);
    }
    return (!low || ord2f(*(volatile const int *)&st->vs.vmin) == mn) && (!high || ord2f(*(volatile const int *)&st->vs.vmax) == mx);
}

// Pass B: undecided voxels get their exact value (and join the bbox if >= iso);
// the range is the exact extreme over the candidates of k_od_scan.  Where those are more
// than a list holds, OD_SAMPLE of them are looked at, and their extreme is the volume's if it
// is the bound that the raw volume gives (plateau_holds): so for a constant background
// or a saturated region, which has voxels whose whole window is that value.  Else the caller
// falls back.  The constant background of a skull-stripped head or of a padded CT fell back on
// every call without this: 181 x 217 x 181 head 337 -> 284 us (604 -> 414 labelled),
// 511 x 512 x 300 CT 1619 -> 1079 (2330 -> 1258).  A warp per
// voxel: 25 lanes take one row's x tap each, five the y taps, then the z tap, all in
// the reference's double sequence (a thread per voxel walked the 31 taps one after
// another: 29 us for the 512^3 CT volume's few thousand voxels).
__global__ void __launch_bounds__(256) k_od_resolve(const float *__restrict__ in, float *out, int nx, int ny, int nz,
                                                    float iso, OdStats *st, OdLists L, bool at_or_above) {
    grid_wait();
    const unsigned FULL = 0xffffffffu;
    const bool low = st->cnt[1] > L.cap, high = st->cnt[2] > L.cap;   // lists that do not hold every candidate
    const unsigned nu = st->cnt[0], nmin = low ? OD_SAMPLE : st->cnt[1], nmax = high ? OD_SAMPLE : st->cnt[2], n = nu + nmin + nmax;
    const unsigned flags = st->flags;
    if (flags || nu > L.cap || !nmin || !nmax) {   // the caller falls back
        if (blockIdx.x == 0 && threadIdx.x == 0) od_flag(st, OD_FALLBACK);
        return;
    }
    const int lane = threadIdx.x & 31;
    const unsigned every = L.cap / OD_SAMPLE;
    for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {
        const int which = i < nu ? 0 : (i < nu + nmin ? 1 : 2);
        const unsigned k1 = i - nu, k2 = k1 - nmin;
        const unsigned j = which == 0 ? L.unc[i] : (which == 1 ? L.cmin[low ? k1 * every : k1] : L.cmax[high ? k2 * every : k2]);
        const unsigned q = j / (unsigned)nx;
        const int x = (int)(j - q * (unsigned)nx), z = (int)(q / (unsigned)ny), y = (int)(q - (unsigned)z * (unsigned)ny);
        const bool xi = x >= 2 && x <= nx - 3, yi = y >= 2 && y <= ny - 3, zi = z >= 2 && z <= nz - 3;
        // lane 5 * dz + dy: the x value of row (y - 2 + dy, z - 2 + dz); rows past the volume are not used
        const int yy = y - 2 + lane % 5, zz = z - 2 + lane / 5;
        float X = 0.f;
        if (lane < 25 && yy >= 0 && yy < ny && zz >= 0 && zz < nz) {
            const float *p = in + ((size_t)zz * ny + yy) * nx + x;
            X = xi ? tap5_double(p[-2], p[-1], p[0], p[1], p[2]) : p[0];
        }
        const int r = min(lane, 4) * 5;
        const float a = __shfl_sync(FULL, X, r), b = __shfl_sync(FULL, X, r + 1), c = __shfl_sync(FULL, X, r + 2),
                    d = __shfl_sync(FULL, X, r + 3), e = __shfl_sync(FULL, X, r + 4);
        const float Y = lane < 5 && yi ? tap5_double(a, b, c, d, e) : c;
        const float f = __shfl_sync(FULL, Y, 0), g = __shfl_sync(FULL, Y, 1), h = __shfl_sync(FULL, Y, 2),
                    k = __shfl_sync(FULL, Y, 3), l = __shfl_sync(FULL, Y, 4);
        if (lane != 0) continue;
        const float v = zi ? tap5_double(f, g, h, k, l) : h;
        if (which == 0) {
            out[j] = v;
            unsigned *sw = L.vsign + od_vsign_word((unsigned)x, (unsigned)y, (unsigned)z, L.wv, L.nys);
            if (at_or_above ? v >= iso : __fsub_rn(v, iso) > -N2M_FLT_EPS) atomicOr(sw, 1u << (x & 31));
            else atomicAnd(sw, ~(1u << (x & 31)));
            if (v >= iso) {
                atomicMin(&st->vs.lo[0], x); atomicMax(&st->vs.hi[0], x);
                atomicMin(&st->vs.lo[1], y); atomicMax(&st->vs.hi[1], y);
                atomicMin(&st->vs.lo[2], z); atomicMax(&st->vs.hi[2], z);
            }
        } else if (which == 1) {
            atomicMin(&st->vs.vmin, f2ord(v));
        } else {
            atomicMax(&st->vs.vmax, f2ord(v));
        }
    }
    if (!low && !high) return;
    raw_extremes(in, nx, ny, nz, st);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&st->done, 1u) == gridDim.x - 1) {   // the last block
        __threadfence();
        if (!plateau_holds(st, low, high)) od_flag(st, OD_FALLBACK);
    }
}

// ---- marks -> the exact passes on marked voxels ----------------------------------
// The words of marked voxels (whose z outputs are wanted), of the voxels whose y values
// those need (+-2 slices) and of the voxels whose x values those need (+-2 rows), each
// as a list of {voxel of bit 0, bits}.  A block takes OL_T words of OL_Z slices of the
// row-aligned mark bitmap: the y marks of its words and of two rows either way go to
// shared memory (a window of five slices slides along z: one load per word and slice
// and four more per run), the x marks are five of those; one atomic per list and block
// reserves the room (the lists' order is free).
// 512^3: 24 us; listing voxels instead of words took 81 us and 250 MB of list traffic,
// two dilations, a scan over every word and a scatter 180 us.
constexpr int OL_T = 256, OL_Z = 8, OL_MAXW = 64;   // rows of more than OL_MAXW words read their halo from global memory

__device__ __forceinline__ unsigned y_marks(const unsigned *__restrict__ need, unsigned i, unsigned slice, int z, int nz) {
    unsigned m = 0;
#pragma unroll
    for (int d = -2; d <= 2; d++)
        if (z + d >= 0 && z + d < nz) m |= __ldg(need + (size_t)(z + d) * slice + i);
    return m;
}

__global__ void __launch_bounds__(OL_T) k_od_lists(const unsigned *__restrict__ need, int nx, int nz, unsigned W, unsigned slice,
                                                   unsigned *cnt, uint2 *lz, uint2 *ly, uint2 *lx) {
    grid_wait();
    __shared__ unsigned ym[OL_Z][OL_T + 4 * OL_MAXW];
    __shared__ unsigned wsum[3][OL_T / 32], base[3];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned bps = (slice + OL_T - 1) / OL_T;   // blocks per slice
    const int z0 = (int)(blockIdx.x / bps) * OL_Z;
    const unsigned i0 = blockIdx.x % bps * OL_T, i = i0 + (unsigned)tid;
    const bool in = i < slice;
    unsigned mx[OL_Z], my[OL_Z], mz[OL_Z], any = 0u;
    if (W <= (unsigned)OL_MAXW) {
        const int h = 2 * (int)W;   // halo words either side
        for (int k = tid; k < OL_T + 2 * h; k += OL_T) {
            const long long q = (long long)i0 + k - h;
            unsigned v[OL_Z + 4];
#pragma unroll
            for (int d = 0; d < OL_Z + 4; d++) {
                const int z = z0 - 2 + d;
                v[d] = q >= 0 && q < (long long)slice && z >= 0 && z < nz ? __ldg(need + (size_t)z * slice + (size_t)q) : 0u;
            }
#pragma unroll
            for (int d = 0; d < OL_Z; d++) {
                ym[d][k] = z0 + d < nz ? v[d] | v[d + 1] | v[d + 2] | v[d + 3] | v[d + 4] : 0u;
                any |= ym[d][k];
            }
        }
        if (!__syncthreads_or(any != 0u)) return;
#pragma unroll
        for (int d = 0; d < OL_Z; d++) {
            my[d] = in ? ym[d][tid + h] : 0u;
            mx[d] = 0u;
#pragma unroll
            for (int e = 0; e <= 4; e++) mx[d] |= ym[d][tid + e * (int)W];
            if (!in) mx[d] = 0u;
        }
    } else {
#pragma unroll
        for (int d = 0; d < OL_Z; d++) {
            my[d] = in && z0 + d < nz ? y_marks(need, i, slice, z0 + d, nz) : 0u;
            mx[d] = my[d];
            for (int e = -2; e <= 2; e++) {
                const long long q = (long long)i + (long long)e * W;
                if (e && in && z0 + d < nz && q >= 0 && q < (long long)slice) mx[d] |= y_marks(need, (unsigned)q, slice, z0 + d, nz);
            }
            any |= mx[d];
        }
        if (!__syncthreads_or(any != 0u)) return;
    }
    unsigned c[3] = {0u, 0u, 0u};   // this warp's words in each list
#pragma unroll
    for (int d = 0; d < OL_Z; d++) {
        mz[d] = my[d] ? __ldg(need + (size_t)(z0 + d) * slice + i) : 0u;
        c[0] += __popc(__ballot_sync(FULL, mz[d] != 0u));
        c[1] += __popc(__ballot_sync(FULL, my[d] != 0u));
        c[2] += __popc(__ballot_sync(FULL, mx[d] != 0u));
    }
    if (lane == 0)
        for (int l = 0; l < 3; l++) wsum[l][wid] = c[l];
    __syncthreads();
    if (tid < 3) {
        unsigned t = 0;
        for (int k = 0; k < OL_T / 32; k++) t += wsum[tid][k];
        base[tid] = t ? atomicAdd(cnt + tid, t) : 0u;
    }
    __syncthreads();
    unsigned at[3];
#pragma unroll
    for (int l = 0; l < 3; l++) {
        at[l] = base[l];
        for (int k = 0; k < wid; k++) at[l] += wsum[l][k];
    }
    const unsigned ny = slice / W, row = i / W, lt = (1u << lane) - 1u;
    unsigned v0 = ((unsigned)z0 * ny + row) * (unsigned)nx + (i - row * W) * 32u;
    auto write = [&](unsigned m, unsigned &o, uint2 *list) {
        const unsigned b = __ballot_sync(FULL, m != 0u);
        if (m) list[o + __popc(b & lt)] = make_uint2(v0, m);
        o += __popc(b);
    };
#pragma unroll
    for (int d = 0; d < OL_Z; d++) {
        write(mz[d], at[0], lz);
        write(my[d], at[1], ly);
        write(mx[d], at[2], lx);
        v0 += ny * (unsigned)nx;
    }
}

// one exact pass on the listed voxels: dst[v] = tap sum of src along the axis
// (AXIS 0, 1, 2: x, y, z), or src[v] on the two face layers.  A warp takes 32 listed
// words, writes their voxels as a dense list in shared memory and works through it,
// OE_U voxels per lane in flight at once; undecided taps queued per warp for the
// FP64 fix-up.  Bound by the gathers' latency and instruction issue: the x, y and z passes
// of the 512^3 CT volume take 92, 91 and 70 us.
constexpr int OE_U = 4, OE_T = 128;
template <int AXIS>
__global__ void __launch_bounds__(OE_T, 10) k_od_exact(const uint2 *__restrict__ list, const unsigned *__restrict__ cnt,
                                                   const float *__restrict__ src, float *dst, unsigned nx, unsigned ny, unsigned nz,
                                                   unsigned long long mnx, unsigned long long mny) {
    grid_wait();
    __shared__ unsigned stage_buf[OE_T / 32][32 * (OE_U + 1)];   // < 32 between drains, + 32 per entry
    __shared__ unsigned short item[OE_T / 32][32 * 32];          // word << 5 | bit
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    FixStage<false> F{stage_buf[wid], 0};
    Acc acc;   // unused
    const unsigned stride = AXIS == 0 ? 1u : (AXIS == 1 ? nx : nx * ny);
    const Pass P{src, dst, stride, 0, 0, 0u, 0.f, nullptr};
    const unsigned n = *cnt, warps = gridDim.x * OE_T / 32u;
    // words of a warp at a time: fewer when the list is too short to give every warp 32
    const unsigned per = n >= 64u * warps ? 32u : (n >= 16u * warps ? 16u : (n >= 4u * warps ? 8u : 4u));
    for (unsigned i0 = ((blockIdx.x * OE_T + threadIdx.x) >> 5) * per; i0 < n; i0 += warps * per) {   // warp-uniform
        const uint2 e = (unsigned)lane < per && i0 + (unsigned)lane < n ? __ldg(list + i0 + lane) : make_uint2(0u, 0u);
        // x of bit 0, or whether the word's row (slice) is two rows (slices) away from the faces
        const unsigned row = nx == 1u ? e.x : (unsigned)__umul64hi(e.x, mnx);   // e.x / nx
        const unsigned sl = ny == 1u ? row : (unsigned)__umul64hi(row, mny);    // row / ny
        const unsigned c0 = AXIS == 0 ? e.x - row * nx : (AXIS == 1 ? row - sl * ny : sl);
        const unsigned len = AXIS == 0 ? nx : (AXIS == 1 ? ny : nz);
        const bool winner = c0 >= 2u && c0 + 2u < len;
        unsigned total;
        {
            unsigned incl = __popc(e.y);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned t = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += t;
            }
            total = __shfl_sync(FULL, incl, 31);
            unsigned at = incl - __popc(e.y);
            for (unsigned m = e.y; m; m &= m - 1u) item[wid][at++] = (unsigned short)(lane << 5 | (__ffs(m) - 1));
        }
        __syncwarp();
        for (unsigned k0 = 0; k0 < total; k0 += 32u * OE_U) {
            unsigned v[OE_U];
            bool act[OE_U], inner[OE_U];
            float a[OE_U][5];
#pragma unroll
            for (int u = 0; u < OE_U; u++) {
                const unsigned k = k0 + (unsigned)u * 32u + (unsigned)lane;
                act[u] = k < total;
                const unsigned it = act[u] ? item[wid][k] : 0u, b = it & 31u;
                v[u] = __shfl_sync(FULL, e.x, (int)(it >> 5)) + b;
                if (AXIS == 0) {
                    const unsigned x = __shfl_sync(FULL, c0, (int)(it >> 5)) + b;
                    inner[u] = act[u] && x >= 2u && x + 2u < len;
                } else {
                    inner[u] = __shfl_sync(FULL, winner, (int)(it >> 5)) && act[u];
                }
                const float *p = src + v[u];
                if (inner[u]) {
                    a[u][0] = __ldg(p - 2 * (size_t)stride);
                    a[u][1] = __ldg(p - (size_t)stride);
                    a[u][3] = __ldg(p + stride);
                    a[u][4] = __ldg(p + 2 * (size_t)stride);
                }
                a[u][2] = act[u] ? __ldg(p) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < OE_U; u++) {
                bool fail = false;
                if (act[u]) {
                    float r = a[u][2];
                    // undecided by the split: nearly always an exact tie, which tap5_fast cannot decide either
                    if (inner[u]) {
                        const int q = tap5_split_state(a[u][0], a[u][1], a[u][2], a[u][3], a[u][4], &r);
                        fail = q < 0 ? !tap5_fast(a[u][0], a[u][1], a[u][2], a[u][3], a[u][4], &r) : q == 0;
                    }
                    if (!fail) dst[v[u]] = r;
                }
                F.push(fail, v[u], lane);
            }
            F.drain(P, acc, lane);
        }
        __syncwarp();   // the item list is reused
    }
    F.finish(P, acc, lane);
}

// the labelling's effect on the exact values the z pass just wrote at the listed words' voxels
__global__ void __launch_bounds__(256) k_od_post(const uint2 *__restrict__ list, const unsigned *__restrict__ cnt, float *out,
                                                 LabelPost L, int nx, int ny) {
    grid_wait();
    const unsigned n = *cnt;
    const int lane = threadIdx.x & 31;
    for (unsigned i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += (gridDim.x * blockDim.x) >> 5) {   // a warp per word
        const uint2 e = list[i];
        const unsigned row = e.x / (unsigned)nx;
        const size_t w = (size_t)row * L.W + ((e.x - row * (unsigned)nx) >> 5);
        const unsigned kept = L.K[w], kd = L.KD[w];
        if (!(e.y >> lane & 1u)) continue;
        float *v = out + e.x + (unsigned)lane;
        if (!(kd >> lane & 1u)) *v = L.mn;
        else if (L.fill && (kept >> lane & 1u)) *v = fmaxf(*v, L.iso);
    }
}

// floor(2^64 / d) + 1: __umul64hi(n, m) = n / d for every 32-bit n (d >= 2)
unsigned long long od_magic(unsigned d) { return d <= 1u ? 0ull : ~0ull / d + 1ull; }

int od_grid(const void *fn, int threads) {
    int dev = 0, sms = 0, per_sm = 0, g = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, 0) == cudaSuccess)
        g = sms * std::max(per_sm, 1);
    cudaGetLastError();
    return g > 0 ? g : 152 * 4;
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
        cudaGetLastError();
    });
    return fn;
}
}  // namespace

bool od_eligible(int nx, int ny, int nz) {
    return (size_t)nx * ny * nz < ((size_t)1 << 32) && nx >= 5 && ny >= 5 && nz >= 5;
}

namespace {
bool od_odd(const float *in, int nx) { return nx % 4 != 0 || ((uintptr_t)in & 15u) != 0; }
}  // namespace
size_t od_scratch(const float *in, int nx, int ny, int nz) {
    return (size_t)(od_odd(in, nx) ? (nx + 3) / 4 * 4 : nx) * ny * nz * sizeof(float);
}

namespace {
// rows of nx values with a pitch of px (a multiple of 4), a thread per four
__global__ void __launch_bounds__(256) k_od_pad(const float *__restrict__ in, float *out, int nx, int px, size_t n4) {
    grid_wait();
    for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < n4; i += (size_t)gridDim.x * 256) {
        const unsigned q = (unsigned)px / 4u;
        const size_t row = n4 < ((size_t)1 << 32) ? (size_t)((unsigned)i / q) : i / q;
        const int x = 4 * (int)(i - row * q);
        const float *p = in + row * nx + x;
        float4 v = make_float4(__ldg(p), 0.f, 0.f, 0.f);
        if (x + 1 < nx) v.y = __ldg(p + 1);
        if (x + 2 < nx) v.z = __ldg(p + 2);
        if (x + 3 < nx) v.w = __ldg(p + 3);
        ((float4 *)out)[i] = v;
    }
}

// slices per task: long runs read few slices twice (zrun + 4 for zrun); a volume too
// small to give every warp of the GPU a task takes shorter ones instead (64^3: 45 us
// with 32 slices per task for want of warps)
int od_zrun(int nx, int ny, int nz) {
    const long long cols = (long long)((nx + OA_X - 1) / OA_X) * ((ny + OA_Y - 1) / OA_Y);
    int zrun = 32;
    while (zrun > 4 && cols * ((nz + zrun - 1) / zrun) < 152 * 8) zrun /= 2;
    return zrun;
}
// warp tasks of pass A
size_t od_tasks(int nx, int ny, int nz, int zrun) {
    return (size_t)((nx + OA_X - 1) / OA_X) * ((ny + OA_Y - 1) / OA_Y) * ((nz + zrun - 1) / zrun);
}
constexpr size_t OD_LISTS = (sizeof(OdStats) + 255) / 256 * 256;   // where the lists begin behind the statistics
OdLists od_lists(const OdWork &w, int nx, int ny) {
    unsigned *const unc = (unsigned *)((char *)w.st.p + OD_LISTS);   // three lists, then the ranges
    return OdLists{unc, unc + w.cap, unc + 2 * (size_t)w.cap,
                   (unsigned *)((char *)w.st.p + offsetof(OdStats, cnt)), w.cap, w.vsign.as<unsigned>(), (float4 *)(unc + 3 * (size_t)w.cap),
                   (unsigned)(nx + 31) / 32, (unsigned)(ny + 7) / 8};
}
}  // namespace

n2m_status od_approx(const float *in, float *out, int nx, int ny, int nz, float iso, float *scratch, OdWork &w, cudaStream_t s) {
    const size_t n = (size_t)nx * ny * nz;
    auto encode = tensor_map_encoder();
    if (!encode) {
        n2m_set_error("cuTensorMapEncodeTiled is not available from the driver");
        return N2M_ERR_CUDA;
    }
    const bool odd = od_odd(in, nx) || ((uintptr_t)out & 15u) != 0;
    const int px = (nx + 3) / 4 * 4;
    const float *rows = in;
    if (odd) {
        const size_t n4 = (size_t)px / 4 * ny * nz;
        n2m_launch(k_od_pad, (unsigned)std::min<size_t>((n4 + 255) / 256, 152u * 32u), 256, 0, s, in, scratch, nx, px, n4);
        rows = scratch;
    }
    CUtensorMap tmap;
    {
        const cuuint64_t gdim[3] = {(cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
        const cuuint64_t gstride[2] = {(cuuint64_t)px * 4u, (cuuint64_t)px * ny * 4u};
        const cuuint32_t box[3] = {OA_BW, OA_BH, 1}, estr[3] = {1, 1, 1};
        const CUresult r = encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void *)rows, gdim, gstride, box, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                  CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) {
            n2m_set_error("cuTensorMapEncodeTiled failed (%d)", (int)r);
            return N2M_ERR_CUDA;
        }
    }
    w.cap = (unsigned)std::min<size_t>(n / 64 + OD_SAMPLE, 1u << 22) & ~3u;   // the ranges behind the lists stay aligned
    const int zrun = od_zrun(nx, ny, nz);
    const size_t nys = (size_t)(ny + 7) / 8, wv = (size_t)(nx + 31) / 32, ntask = od_tasks(nx, ny, nz, zrun);
    CKS(w.st.ensure(OD_LISTS + 3 * (size_t)w.cap * sizeof(unsigned) + ntask * sizeof(float4)));
    CKS(w.vsign.ensure((size_t)nz * nys * wv * 8 * sizeof(unsigned)));
    OdStats h{};
    stats_init_host(&h.vs);   // vmin / vmax are filled by pass B from the candidates
    h.umin = INT_MAX;
    h.lmax = INT_MIN;
    for (int c = 0; c < 4; c++) {
        h.rlo[c] = INT_MAX;
        h.rhi[c] = INT_MIN;
    }
    CK(cudaMemcpyAsync(w.st.p, &h, sizeof(OdStats), cudaMemcpyHostToDevice, s));
    const auto approx = odd ? k_od_approx<true> : k_od_approx<false>;
    const unsigned grid = (unsigned)std::min<size_t>((ntask + OA_WARPS - 1) / OA_WARPS, (size_t)od_grid((const void *)approx, OA_WARPS * 32));
    n2m_launch(approx, grid, OA_WARPS * 32, 0, s, tmap, out, nx, ny, nz, zrun, iso, w.st.as<OdStats>(), od_lists(w, nx, ny));
    CKL();
    return N2M_OK;
}

n2m_status od_resolve(const float *in, float *out, int nx, int ny, int nz, float iso, OdWork &w, cudaStream_t s,
                      bool at_or_above) {
    const OdLists L = od_lists(w, nx, ny);
    const int zrun = od_zrun(nx, ny, nz);
    const size_t ntask = od_tasks(nx, ny, nz, zrun);
    n2m_launch(k_od_scan, (unsigned)((ntask + OS_T - 1) / OS_T), 256, 0, s, out, nx, ny, nz, zrun, w.st.as<OdStats>(), L);
    n2m_launch(k_od_resolve, 152 * 8, 256, 0, s, in, out, nx, ny, nz, iso, w.st.as<OdStats>(), L, at_or_above);
    CKL();
    return N2M_OK;
}

n2m_status od_check(const OdStats &h, bool *fallback) {
    if (h.flags & OD_TIMEOUT) {
        n2m_set_error("pre-smooth: a tile copy did not complete");
        return N2M_ERR_TIMEOUT;
    }
    *fallback = (h.flags & OD_FALLBACK) != 0;
    return N2M_OK;
}

n2m_status od_marks(OdWork &w, const int dim[3], unsigned **need, cudaStream_t s) {
    const size_t bytes = (size_t)((dim[0] + 31) / 32) * dim[1] * dim[2] * sizeof(unsigned);
    CKS(w.need.ensure(bytes));
    CK(cudaMemsetAsync(w.need.p, 0, bytes, s));
    *need = w.need.as<unsigned>();
    return N2M_OK;
}

n2m_status od_repair(const OdRepair &r, cudaStream_t s) {
    OdWork &w = *r.w;
    const int nx = r.dim[0], ny = r.dim[1], nz = r.dim[2];
    const unsigned W = (unsigned)(nx + 31) / 32u, slice = W * (unsigned)ny, bps = (slice + OL_T - 1) / OL_T;
    const size_t nw = (size_t)slice * nz;
    CKS(w.list.ensure(3 * nw * sizeof(uint2)));   // every list fits any marking
    CKS(w.lcnt.ensure(sizeof(uint4)));
    unsigned *cnt = w.lcnt.as<unsigned>();   // z, y, x counts
    uint2 *lz = w.list.as<uint2>(), *ly = lz + nw, *lx = ly + nw;
    CK(cudaMemsetAsync(cnt, 0, sizeof(uint4), s));
    n2m_launch(k_od_lists, bps * (unsigned)((nz + OL_Z - 1) / OL_Z), OL_T, 0, s, w.need.as<unsigned>(), nx, nz, W, slice, cnt,
               lz, ly, lx);
    CKL();
    const int xb = od_grid((const void *)k_od_exact<0>, OE_T);
    const unsigned ux = (unsigned)nx, uy = (unsigned)ny, uz = (unsigned)nz;
    const unsigned long long mx = od_magic(ux), my = od_magic(uy);
    n2m_launch(k_od_exact<0>, xb, OE_T, 0, s, lx, cnt + 2, r.in, r.tmp1, ux, uy, uz, mx, my);
    n2m_launch(k_od_exact<1>, xb, OE_T, 0, s, ly, cnt + 1, r.tmp1, r.tmp2, ux, uy, uz, mx, my);
    n2m_launch(k_od_exact<2>, xb, OE_T, 0, s, lz, cnt + 0, r.tmp2, r.out, ux, uy, uz, mx, my);
    if (r.post) n2m_launch(k_od_post, 152 * 8, 256, 0, s, lz, cnt + 0, r.out, *r.post, nx, ny);
    CKL();
    return N2M_OK;
}
