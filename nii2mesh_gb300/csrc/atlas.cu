// atlas.cu — batched atlas meshing (the per-label loop of src/nii2mesh.c:492-583).
//
// The reference binarises the whole volume for every label (`lo < v < hi`,
// src/nii2mesh.c:555-563) and runs the full meshify on it.  Outside the
// label's bounding box + 2 voxels the smoothed mask is exactly 0, so every
// stage can run on a sub-box (bbox + 3, clipped to the volume) instead:
// smoothing keeps the volume's own face rule (global coordinates), the
// background outside the sub-box joins the sub-box's boundary shell (so
// bubble detection and the largest-cluster tie-break are unchanged), and the
// marching-cubes fetch returns 0 for voxels outside the sub-box.
//
// All labels' sub-boxes live in one float arena, and their rows in one array of bit words
// (a box begins at a multiple of 32 words).  Each stage is one launch over the words,
// runs or points of every box, so hundreds of labels of very different sizes share the GPU
// in each launch.  The masks are smoothed from their bits, the components are found on
// runs listed across the boxes, the clustered values are never written (their signs follow
// from the kept set, agval applies the rest where marching cubes reads), and the
// boxes' grids are words of one numbering for the kernels of mcwords.cuh: each label's
// mesh is a contiguous range in the concatenated output, numbered exactly as the
// single-volume path.  256^3 atlas of 250 labels: 3834 us when every stage went over the
// voxels or rows of the arena, 1804 us now.
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "mc33.cuh"
#include "mcwords.cuh"
#include "runs.cuh"
#include "smooth_core.cuh"
#include "uf.cuh"

namespace {
using namespace mc33;
using namespace runs;

struct ABox {
    int label;
    int o[3], n[3];            // sub-box origin and size (global voxel coordinates)
    long long arena;           // arena offset of the sub-box
    unsigned tile0;            // first smoothing unit of this box
    int full;                  // sub-box covers the whole volume
    int fail;                  // N2M status of this label (0 = ok)
    int vmin, vmax;            // ordered-int range of the smoothed sub-box
    int amin;                  // ordered-int min after clustering
    float iso, edge_max, pad;
    int blo[3], bhi[3];        // bbox of voxels >= iso (global)
    unsigned nbg, nfg;         // component counts
    unsigned long long best;   // largest component (size << 32 | ~root)
    // marching-cubes grid (global origin lo, size gn), filled by the host
    int glo[3], gn[3];
    unsigned WX, word0;
    // bit words per row, first bit word across the boxes
    unsigned W, bw0;
};

struct AtlasVol {
    const short *lab;
    int nx, ny, nz;
    long long nxy, nvox;
};

__device__ __forceinline__ int find_item(const ABox *b, int nb, unsigned item, unsigned ABox::*field) {
    int lo = 0, hi = nb - 1;
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (b[m].*field <= item) lo = m;
        else hi = m - 1;
    }
    return lo;
}

// ---- S0: every label's bounding box and the largest label -------------------------
// A thread takes HV consecutive voxels of a row, loaded at once.  Atomics on a label's box
// are the bound (a label's rows come in order, so nearly every run moves its box on, and a
// few hundred boxes are a few dozen cache lines): the lanes of a warp whose runs have the
// same label agree on one extent, a block keeps the boxes of its consecutive rows in shared
// memory, and sends them on where they exceed the box as last seen (boxes only grow: an old
// view is safe).  256^3: 259 us with a thread per 32 voxels and seven global atomics for every
// run, 234 us without the blocks' tables, 79 us now.
constexpr int HV = 8, HT = 256;   // voxels of a thread, entries of a block's table
__device__ __forceinline__ void grow_box(int *b, int x0, int x1, int y0, int y1, int z0, int z1) {
    volatile int *seen = b;
    const int b0 = seen[0], b1 = seen[1], b2 = seen[2], b3 = seen[3], b4 = seen[4], b5 = seen[5];
    if (x0 < b0) atomicMin(b, x0);
    if (y0 < b1) atomicMin(b + 1, y0);
    if (z0 < b2) atomicMin(b + 2, z0);
    if (x1 > b3) atomicMax(b + 3, x1);
    if (y1 > b4) atomicMax(b + 4, y1);
    if (z1 > b5) atomicMax(b + 5, z1);
}
__global__ void __launch_bounds__(HT) k_a_hist(AtlasVol v, int maxlab, unsigned *present, int *bb, int *vmax) {
    grid_wait();
    int mx = 0;
    const unsigned spr = (unsigned)(v.nx + HV - 1) / HV, lane = threadIdx.x & 31u;
    const unsigned long long nseg = (unsigned long long)spr * v.ny * v.nz, nseg32 = (nseg + 31) & ~31ull;
    const bool vec = v.nx % HV == 0 && ((size_t)v.lab & 15) == 0, small = nseg32 < 0x80000000ull;   // cheap divisions
    __shared__ int key[HT], box[HT][6];
    key[threadIdx.x] = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) box[threadIdx.x][k] = k < 3 ? INT_MAX : INT_MIN;
    __syncthreads();
    const unsigned long long per = ((nseg32 + gridDim.x - 1) / gridDim.x + 31) & ~31ull, s0 = per * blockIdx.x;
    const unsigned long long s1 = min(nseg32, s0 + per);
    for (unsigned long long sg = s0 + threadIdx.x; sg < s1; sg += HT) {   // whole warps
        const unsigned row = small ? (unsigned)sg / spr : (unsigned)(sg / spr);
        const int xs = (int)(sg - (unsigned long long)row * spr) * HV, n = sg < nseg ? min(HV, v.nx - xs) : 0;
        const int z = (int)(row / (unsigned)v.ny), y = (int)(row - (unsigned)z * (unsigned)v.ny);
        const short *p = v.lab + (long long)row * v.nx + xs;
        short l[HV];
        if (vec && n) {
            *(int4 *)l = __ldg((const int4 *)p);
        } else {
#pragma unroll
            for (int k = 0; k < HV; k++) l[k] = k < n ? p[k] : (short)0;
        }
        unsigned ends = 0;   // last voxels of runs of labels
#pragma unroll
        for (int k = 0; k < HV; k++) {
            mx = max(mx, (int)l[k]);
            if (l[k] > 0 && (int)l[k] <= maxlab && (k == HV - 1 || l[k + (k < HV - 1)] != l[k])) ends |= 1u << k;
        }
        unsigned done = 0;   // voxels of runs already sent
        while (__any_sync(FULL, ends != 0u)) {
            int lab = 0, first = 0, last = 0;
            if (ends) {
                const int e = __ffs(ends) - 1;
#pragma unroll
                for (int k = 0; k < HV; k++)
                    if (k == e) lab = l[k];
                first = e;
#pragma unroll
                for (int k = HV - 2; k >= 0; k--)
                    if (k < first && k == first - 1 && !(done >> k & 1u) && l[k] == lab) first = k;
                last = xs + e;
                done |= (2u << e) - 1u;
                first += xs;
                ends &= ends - 1u;
            }
            const unsigned peers = __match_any_sync(FULL, lab);
            const int x0 = __reduce_min_sync(peers, first), x1 = __reduce_max_sync(peers, last);
            const int y0 = __reduce_min_sync(peers, y), y1 = __reduce_max_sync(peers, y);
            const int z0 = __reduce_min_sync(peers, z), z1 = __reduce_max_sync(peers, z);
            if (lab && lane == (unsigned)__ffs(peers) - 1u) {
                int at = -1;
                for (int t = 0; t < 4 && at < 0; t++) {
                    const int i = (lab + 61 * t) & (HT - 1), had = atomicCAS(&key[i], 0, lab);
                    if (had == 0 || had == lab) at = i;
                }
                if (at >= 0) {
                    grow_box(box[at], x0, x1, y0, y1, z0, z1);
                } else {
                    grow_box(bb + 6 * lab, x0, x1, y0, y1, z0, z1);
                    present[lab] = 1u;
                }
            }
        }
    }
    __shared__ int bmx;
    if (threadIdx.x == 0) bmx = 0;
    __syncthreads();
    mx = __reduce_max_sync(FULL, mx);
    if ((threadIdx.x & 31) == 0) atomicMax(&bmx, mx);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(vmax, bmx);
    if (const int lab = key[threadIdx.x]) {
        const int *b = box[threadIdx.x];
        grow_box(bb + 6 * lab, b[0], b[3], b[1], b[4], b[2], b[5]);
        present[lab] = 1u;
    }
}

// ---- S1: binarise + pre-smooth every sub-box -----------------------------------------
// The boxes' rows are bit words (bit x & 31 of word B.bw0 + (z*n1 + y)*B.W + x/32, local
// coordinates; a box begins at a multiple of 32 words, the filling is zero), and a warp
// takes 32 words of one box at a time.
struct WordAt {
    unsigned lr;   // local row
    int w;         // word of the row
    bool live;
};
__device__ __forceinline__ WordAt word_at(const ABox &B, unsigned lw) {
    WordAt a;
    a.lr = lw / B.W;
    a.w = (int)(lw - a.lr * B.W);
    a.live = a.lr < (unsigned)B.n[1] * (unsigned)B.n[2];
    return a;
}
// bits of the 32 words of a warp, AW_U words in flight: off(row) is where a row's values begin in p (found once per
// word, by its own lane), bit(value) decides
constexpr int AW_U = 16;
template <class V, class O, class P>
__device__ __forceinline__ unsigned warp_words(const ABox &B, unsigned lw0, int lane, const V *__restrict__ p, O off, P bit) {
    const WordAt a = word_at(B, lw0 + (unsigned)lane);
    const int n = __popc(__ballot_sync(FULL, a.live)), left = B.n[0] - 32 * a.w;   // columns from the word's first on
    const long long at = a.live ? off(a.lr) + 32 * a.w : 0;
    unsigned mine = 0;
    for (int k0 = 0; k0 < n; k0 += AW_U) {
        V val[AW_U];
        bool in[AW_U];
#pragma unroll
        for (int u = 0; u < AW_U; u++) {
            const long long q = __shfl_sync(FULL, at, (k0 + u) & 31);
            in[u] = k0 + u < n && lane < __shfl_sync(FULL, left, (k0 + u) & 31);
            val[u] = in[u] ? __ldg(p + q + lane) : V(0);
        }
#pragma unroll
        for (int u = 0; u < AW_U; u++) {
            const unsigned m = __ballot_sync(FULL, in[u] && bit(val[u]));
            if (lane == k0 + u) mine = m;
        }
    }
    return mine;
}

__global__ void __launch_bounds__(256) k_a_mask(AtlasVol v, const ABox *boxes, int nb, unsigned nbw, unsigned *M,
                                                unsigned *wbox) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    for (unsigned w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; w0 < nbw; w0 += gridDim.x * blockDim.x) {
        const int b = find_item(boxes, nb, w0, &ABox::bw0);
        const ABox &B = boxes[b];
        if (lane == 0) wbox[w0 / 32] = (unsigned)b;   // the box of every 32 words
        const int n1 = B.n[1], label = B.label;
        const short *base = v.lab + (long long)B.o[2] * v.nxy + (long long)B.o[1] * v.nx + B.o[0];
        M[w0 + (unsigned)lane] = warp_words(B, w0 - B.bw0, lane, base, [&](unsigned lr) {
            const int z = (int)(lr / (unsigned)n1), y = (int)(lr - (unsigned)z * (unsigned)n1);
            return (long long)z * v.nxy + (long long)y * v.nx;
        }, [&](short l) { return l == label; });
    }
}

// The three passes on the masks' bits.  A warp takes 32 columns x ARY rows and marches along
// z.  The x pass of a binary row has 32 possible results (a table); the y and z passes prove
// the reference's rounding in FP32 (tap5_fast).  What they cannot prove takes the FP64
// sequence: 0.1 % of the y results at once, 1 % of the z results through a queue that
// fills warps (FP64 issues at a 32nd of the FP32 rate).  Slices whose rows are empty, or
// full away from the volume's faces, skip the passes.  Bound by FP32 issue.  23 M arena
// voxels (250 labels of a 256^3 atlas): 604 us with one CTA per column tile, staging and
// queueing every pass between barriers; 200 us.
constexpr int ARY = 4, AZC = 24, AWARPS = 8;
struct SmoothQueue {
    float v[5][64];
    unsigned at[64];
};
__global__ void __launch_bounds__(32 * AWARPS) k_a_smooth(ABox *boxes, int nb, unsigned nunits, const unsigned *__restrict__ M,
                                                          float *arena, int nx, int ny, int nz, bool smooth_on) {
    grid_wait();
    __shared__ float lut[32];
    __shared__ SmoothQueue queues[AWARPS];
    const int lane = threadIdx.x & 31;
    auto tap = [](float a, float b, float c, float d, float e) {
        float r;
        if (!tap5_fast(a, b, c, d, e, &r)) r = tap5_double(a, b, c, d, e);
        return r;
    };
    if (threadIdx.x < 32)
        lut[lane] = tap((float)(lane & 1), (float)(lane >> 1 & 1), (float)(lane >> 2 & 1), (float)(lane >> 3 & 1), (float)(lane >> 4 & 1));
    __syncthreads();
    const float x1 = lut[31], y1 = tap(x1, x1, x1, x1, x1), z1 = tap(y1, y1, y1, y1, y1);   // of a region all ones
    SmoothQueue &q = queues[threadIdx.x >> 5];
    for (unsigned unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; unit < nunits; unit += (gridDim.x * blockDim.x) >> 5) {
        ABox &B = boxes[find_item(boxes, nb, unit, &ABox::tile0)];
        const int n0 = B.n[0], n1 = B.n[1], n2 = B.n[2], W = (int)B.W;
        const unsigned local = unit - B.tile0, ny4 = (unsigned)(n1 + ARY - 1) / ARY;
        const int w = (int)(local % (unsigned)W), y0 = (int)(local / (unsigned)W % ny4) * ARY, z0 = (int)(local / ((unsigned)W * ny4)) * AZC;
        const int zend = min(z0 + AZC, n2), x = 32 * w + lane, gx = B.o[0] + x;
        const bool own = x < n0, xin = gx >= 2 && gx <= nx - 3;
        // no face of the volume within the filter's reach of this unit
        const bool inner = B.o[0] + 32 * w >= 2 && B.o[0] + 32 * w + 31 <= nx - 3 && B.o[1] + y0 >= 2 && B.o[1] + y0 + ARY - 1 <= ny - 3;
        const unsigned *Mb = M + B.bw0;
        float *out = arena + B.arena + x;
        float mn = INFINITY, mx = -INFINITY;
        float r[ARY][5];
#pragma unroll
        for (int k = 0; k < ARY; k++)
#pragma unroll
            for (int t = 0; t < 5; t++) r[k][t] = 0.f;
        unsigned kinds = 0x3ffu, nq = 0;   // the last five slices: 0 empty, 1 full, 2 neither
        auto drain = [&](unsigned n) {     // the queue's first n <= 32
            if ((unsigned)lane < n) {
                const float v = tap5_double(q.v[0][lane], q.v[1][lane], q.v[2][lane], q.v[3][lane], q.v[4][lane]);
                arena[B.arena + q.at[lane]] = v;
                mn = fminf(mn, v);
                mx = fmaxf(mx, v);
            }
            __syncwarp();
        };
        const int zlo = smooth_on ? max(z0 - 2, -B.o[2]) : z0, zhi = smooth_on ? min(zend + 2, nz - B.o[2]) : zend;
        for (int zi = zlo; zi < zhi; zi++) {
            // rows y0-2 .. y0+ARY+1, three words each: lane 3*row + {0, 1, 2}
            unsigned word = 0;
            const int rr = lane / 3, yy = y0 - 2 + rr, ww = w - 1 + lane - 3 * rr;
            if (rr < ARY + 4 && yy >= 0 && yy < n1 && zi >= 0 && zi < n2 && ww >= 0 && ww < W)
                word = __ldg(Mb + ((unsigned)zi * (unsigned)n1 + (unsigned)yy) * (unsigned)W + (unsigned)ww);
            const unsigned prv = __shfl_up_sync(FULL, word, 1), nxt = __shfl_down_sync(FULL, word, 1);
            // at lane 3*row + 1: bits x-2 .. x+33 of the row
            const unsigned lo = word << 2 | prv >> 30, hi = nxt << 2 | word >> 30;
            const bool mid = rr < ARY + 4 && lane - 3 * rr == 1;
            const bool some = __any_sync(FULL, mid && (lo | (hi & 15u)) != 0u);
            const bool all = __all_sync(FULL, !mid || (lo == FULL && (hi & 15u) == 15u));
            const unsigned kind = !smooth_on ? 2u : (!some ? 0u : (all && inner ? 1u : 2u));
            kinds = (kinds << 2 | kind) & 0x3ffu;
            const int gz = B.o[2] + zi, zo = zi - 2, gzo = gz - 2;
            float Y[ARY];
            if (kind == 2u) {
                float xs[ARY + 4];
#pragma unroll
                for (int k = 0; k < ARY + 4; k++) {
                    const unsigned a = __shfl_sync(FULL, lo, 3 * k + 1), b = __shfl_sync(FULL, hi, 3 * k + 1);
                    const unsigned win = __funnelshift_r(a, b, lane) & 31u;
                    xs[k] = smooth_on && xin ? lut[win] : (float)(win >> 2 & 1u);
                }
#pragma unroll
                for (int k = 0; k < ARY; k++) {
                    const int gy = B.o[1] + y0 + k;
                    Y[k] = smooth_on && gy >= 2 && gy <= ny - 3 ? tap(xs[k], xs[k + 1], xs[k + 2], xs[k + 3], xs[k + 4]) : xs[k + 2];
                }
            } else {
#pragma unroll
                for (int k = 0; k < ARY; k++) Y[k] = kind == 0u ? 0.f : y1;
            }
#pragma unroll
            for (int k = 0; k < ARY; k++) {
                r[k][0] = r[k][1]; r[k][1] = r[k][2]; r[k][2] = r[k][3]; r[k][3] = r[k][4]; r[k][4] = Y[k];
            }
            const bool edge = zi >= z0 && zi < zend && (!smooth_on || gz < 2 || gz > nz - 3);   // rows left unfiltered along z
            const bool zint = smooth_on && zo >= z0 && zo < zend && gzo >= 2 && gzo <= nz - 3;
#pragma unroll
            for (int k = 0; k < ARY; k++) {
                if (y0 + k >= n1) break;
                if (edge && own) {
                    out[((long long)zi * n1 + y0 + k) * n0] = Y[k];
                    mn = fminf(mn, Y[k]);
                    mx = fmaxf(mx, Y[k]);
                }
                if (!zint) continue;
                const unsigned at = ((unsigned)zo * (unsigned)n1 + (unsigned)(y0 + k)) * (unsigned)n0;
                float o = 0.f;
                bool ok = true;
                if (kinds == 0x155u) o = z1;
                else if (kinds) ok = tap5_fast(r[k][0], r[k][1], r[k][2], r[k][3], r[k][4], &o);
                if (own && ok) {
                    out[at] = o;
                    mn = fminf(mn, o);
                    mx = fmaxf(mx, o);
                }
                const unsigned fail = __ballot_sync(FULL, own && !ok);
                if (fail) {
                    if (own && !ok) {
                        const unsigned j = nq + __popc(fail & ((1u << lane) - 1u));
#pragma unroll
                        for (int t = 0; t < 5; t++) q.v[t][j] = r[k][t];
                        q.at[j] = at + (unsigned)x;
                    }
                    __syncwarp();
                    nq += __popc(fail);
                    if (nq >= 32) {
                        drain(32);
                        nq -= 32;
                        float mv[5];
                        const unsigned ma = q.at[32 + lane];
#pragma unroll
                        for (int t = 0; t < 5; t++) mv[t] = q.v[t][32 + lane];
                        __syncwarp();
                        if ((unsigned)lane < nq) {
#pragma unroll
                            for (int t = 0; t < 5; t++) q.v[t][lane] = mv[t];
                            q.at[lane] = ma;
                        }
                        __syncwarp();
                    }
                }
            }
        }
        drain(nq);
        for (int o = 16; o; o >>= 1) {
            mn = fminf(mn, __shfl_xor_sync(FULL, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, o));
        }
        if (lane == 0 && mn <= mx) {
            const int a = f2ord(mn), b = f2ord(mx);
            if (a < *(volatile int *)&B.vmin) atomicMin(&B.vmin, a);
            if (b > *(volatile int *)&B.vmax) atomicMax(&B.vmax, b);
        }
    }
}

// ---- S2: per-label isolevel (src/meshify.c:305-321 with iso 0.5) ------------------
__global__ void k_a_iso(ABox *boxes, int nb) {
    grid_wait();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    ABox &B = boxes[b];
    float mn = ord2f(B.vmin), mx = ord2f(B.vmax);
    if (!B.full) mn = fminf(mn, 0.f);   // voxels outside the sub-box are exactly 0
    float iso = 0.5f;
    if (mn == mx) B.fail = N2M_ERR_NO_VARIABILITY;
    if (iso <= mn || iso > mx) iso = (float)(0.5 * (double)__fadd_rn(mn, mx));
    B.iso = iso;
    B.vmin = f2ord(mn);
    B.edge_max = (float)(0.75 * (double)__fadd_rn(mn, iso));
    B.amin = INT_MAX;
}

// ---- S3: clustering on the arena ----------------------------------------------------
// The clustering of label.cu on every sub-box: class masks as bit words, union-find
// links in L (arena-indexed) at the first voxel of each x-run only, boxes independent of
// one another.  The background's face contacts are the box's faces (src/meshify.c:332-336
// on the binarised sub-box).  A warp or a lane per row spent its time on short rows and
// in chains of links (two merges 410 us of the 256^3 atlas, everything else 160); by lists of
// runs and words, links at roots before the merge, all of it takes 330.
__device__ __forceinline__ unsigned ab_valid(const ABox &B, unsigned w) {
    const int x0 = (int)w * 32;
    return x0 + 32 <= B.n[0] ? FULL : (1u << (B.n[0] - x0)) - 1u;
}
// foreground (want 1) or background (want 0) bits of word w of local row lr
__device__ __forceinline__ unsigned ab_class(const unsigned *Bits, const ABox &B, unsigned lr, unsigned w, unsigned want) {
    const unsigned b = Bits[B.bw0 + lr * B.W + w];
    return want ? b : ~b & ab_valid(B, w);
}

// class bits: smoothed value >= the box's isolevel
__global__ void __launch_bounds__(256) k_ab_bits(const ABox *boxes, const unsigned *__restrict__ wbox, unsigned nbw, const float *__restrict__ arena,
                                                 unsigned *Bits) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    for (unsigned w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; w0 < nbw; w0 += gridDim.x * blockDim.x) {
        const ABox &B = boxes[wbox[w0 / 32]];
        const float *base = arena + B.arena;
        const int n0 = B.n[0];
        const float iso = B.iso;
        Bits[w0 + (unsigned)lane] = warp_words(B, w0 - B.bw0, lane, base, [&](unsigned lr) { return (long long)lr * n0; },
                                               [&](float f) { return f >= iso; });
    }
}

// A word of a box's row in a class, with the words before and after it (0 outside the row)
struct AWord {
    unsigned c, pc, nc, lr;
    int w;
    // bits x whose voxel x + dx is in the class
    __device__ __forceinline__ unsigned shifted(int dx) const {
        return dx == 0 ? c : dx == 1 ? (c >> 1) | (nc << 31) : dx == -1 ? (c << 1) | (pc >> 31) : (c << 2) | (pc >> 30);
    }
};
__device__ __forceinline__ AWord aword(const unsigned *__restrict__ Bits, const ABox &B, unsigned lr, int w, unsigned want) {
    return AWord{ab_class(Bits, B, lr, (unsigned)w, want), w ? ab_class(Bits, B, lr, (unsigned)w - 1u, want) : 0u,
                 w + 1 < (int)B.W ? ab_class(Bits, B, lr, (unsigned)w + 1u, want) : 0u, lr, w};
}
// arena index of the start of the run that voxel b (-1 .. 32 of word q) belongs to; rows
// are a few words long, so runs from before the word are walked back
__device__ __forceinline__ int arun(const unsigned *__restrict__ Bits, const ABox &B, unsigned want, const AWord &q, int b) {
    int x = 32 * q.w + 32;
    if (b <= 31 || q.c >> 31) {
        const unsigned z = b < 0 ? 0u : ~q.c & ((1u << min(b, 31)) - 1u);
        x = z ? 32 * q.w + 32 - __clz(z) : 32 * q.w;
        unsigned p = z ? 0u : q.pc;
        for (int w = q.w; p >> 31; p = --w ? ab_class(Bits, B, q.lr, (unsigned)w - 1u, want) : 0u) {
            x = 32 * w - __clz(~p);
            if (~p) break;
        }
    }
    return (int)(B.arena + (long long)q.lr * B.n[0] + x);
}
// the rows before (lr) that touch it: (y-1, z), (y, z-1) and, for 18-connectivity, (y-1, z-1), (y+1, z-1)
template <int NNB> struct ARound {
    static constexpr int NR = NNB == 3 ? 2 : 4, ND = NNB == 3 ? 2 : 8;
    AWord q[NR];
    __device__ __forceinline__ void load(const unsigned *__restrict__ Bits, const ABox &B, unsigned want, unsigned lr, int w) {
        constexpr int RY[4] = {-1, 0, -1, 1}, RZ[4] = {0, -1, -1, -1};
        const int n1 = B.n[1], z = (int)(lr / (unsigned)n1), y = (int)(lr - (unsigned)z * (unsigned)n1);
#pragma unroll
        for (int k = 0; k < NR; k++) {
            const int yy = y + RY[k], zz = z + RZ[k];
            q[k] = yy >= 0 && zz >= 0 && yy < n1 ? aword(Bits, B, (unsigned)(zz * n1 + yy), w, want) : AWord{0u, 0u, 0u, 0u, w};
        }
    }
    // contact directions: the row and the x offset
    static __device__ __forceinline__ constexpr int row(int d) { return d < 2 ? d : d < 4 ? d - 2 + 2 : (d - 4) / 2; }
    static __device__ __forceinline__ constexpr int dx(int d) { return d < 4 ? 0 : (d & 1 ? 1 : -1); }
};

// Run starts of the class as a list {word, arena index}, the words holding any of it as
// another, and every start's link: to the run of its first contact with the rows before
// (without a union), else to itself.  z8 / z32 (may be null) are zeroed there.
constexpr int AL_K = 8;   // words per thread
static_assert(256 * AL_K * 16 < 65536, "a block's run starts and words share one 32-bit sum");
template <int NNB>
__global__ void __launch_bounds__(256) k_al_list(const ABox *boxes, const unsigned *__restrict__ wbox, unsigned nbw,
                                                 const unsigned *__restrict__ Bits, unsigned want, uint2 *list, unsigned *wlist,
                                                 unsigned *n, int *L, unsigned char *z8, unsigned *z32) {
    grid_wait();
    __shared__ unsigned wsum[8], base, wbase;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (unsigned i0 = blockIdx.x * 256 * AL_K; i0 < nbw; i0 += gridDim.x * 256 * AL_K) {
        unsigned st[AL_K], cnt = 0, any = 0;   // run starts | words << 16
#pragma unroll
        for (int k = 0; k < AL_K; k++) {
            const unsigned gw = i0 + (unsigned)(k * 256 + tid);
            st[k] = 0u;
            if (gw < nbw) {
                const ABox &B = boxes[wbox[gw / 32]];
                const WordAt a = word_at(B, gw - B.bw0);
                if (a.live && !B.fail) {
                    const unsigned c = ab_class(Bits, B, a.lr, (unsigned)a.w, want), pc = a.w ? ab_class(Bits, B, a.lr, (unsigned)a.w - 1u, want) : 0u;
                    st[k] = c & ~((c << 1) | (pc >> 31));
                    any |= (c ? 1u : 0u) << k;
                }
            }
            cnt += __popc(st[k]);
        }
        cnt += __popc(any) << 16;
        unsigned incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[wid] = incl;
        __syncthreads();
        if (tid == 0) {
            unsigned t = 0;
            for (int k = 0; k < 8; k++) t += wsum[k];
            if (t) {
                base = atomicAdd(n, t & 0xffffu);
                wbase = atomicAdd(n + 1, t >> 16);
            }
        }
        __syncthreads();
        unsigned before = incl - cnt;
        for (int k = 0; k < wid; k++) before += wsum[k];
        unsigned at = base + (before & 0xffffu), wat = wbase + (before >> 16);
#pragma unroll 1
        for (int k = 0; k < AL_K; k++) {
            if (!(any >> k & 1u)) continue;
            const unsigned gw = i0 + (unsigned)(k * 256 + tid);
            wlist[wat++] = gw;
            unsigned m = 0;   // this word's starts, kept in registers by index above
#pragma unroll
            for (int j = 0; j < AL_K; j++)
                if (j == k) m = st[j];
            if (!m) continue;
            const ABox &B = boxes[wbox[gw / 32]];
            const WordAt a = word_at(B, gw - B.bw0);
            ARound<NNB> A;
            A.load(Bits, B, want, a.lr, a.w);
            const unsigned c = ab_class(Bits, B, a.lr, (unsigned)a.w, want);
            const int row0 = (int)(B.arena + (long long)a.lr * B.n[0] + 32 * a.w);
            for (; m; m &= m - 1) {
                const int b = __ffs(m) - 1, s = row0 + b;
                const unsigned piece = piece_at(c, b);
                int parent = s;
                bool found = false;
#pragma unroll
                for (int d = 0; d < ARound<NNB>::ND; d++) {
                    const unsigned t = piece & A.q[A.row(d)].shifted(A.dx(d));
                    if (!found && t) {
                        found = true;
                        parent = arun(Bits, B, want, A.q[A.row(d)], __ffs(t) - 1 + A.dx(d));
                    }
                }
                list[at++] = make_uint2(gw, (unsigned)s);
                L[s] = parent;
                if (z8) z8[s] = 0;
                if (z32) z32[s] = 0;
            }
        }
        __syncthreads();   // wsum and the bases are reused
    }
}

// Every run start points at its tree's root (links only move to ancestors, which come before
// them, so every walk ends); the way found so far is left for the others.
__global__ void __launch_bounds__(256) k_al_jump(const uint2 *__restrict__ list, const unsigned *__restrict__ n, int *L) {
    grid_wait();
    volatile int *V = L;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < *n; i += gridDim.x * blockDim.x) {
        const int s = (int)list[i].y;
        int p = V[s], at = p, steps = 0;
        for (int q = V[p]; q != p; q = V[p]) {
            p = q;
            if ((++steps & 3) == 0) V[s] = at = p;
        }
        if (p != at) V[s] = p;
    }
}

// Unions, a thread per word of the class: one per overlap of two runs (a contact counts where
// the voxels before it do not also touch), of which nearly all join equal links by now.
template <int NNB>
__global__ void __launch_bounds__(256) k_al_merge(const ABox *boxes, const unsigned *__restrict__ wbox,
                                                  const unsigned *__restrict__ Bits, unsigned want,
                                                  const unsigned *__restrict__ wlist, const unsigned *__restrict__ n, int *L) {
    grid_wait();
    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < n[1]; j += gridDim.x * blockDim.x) {
        const unsigned gw = wlist[j];
        const ABox &B = boxes[wbox[gw / 32]];
        const WordAt at = word_at(B, gw - B.bw0);
        const AWord own = aword(Bits, B, at.lr, at.w, want);
        ARound<NNB> A;
        A.load(Bits, B, want, at.lr, at.w);
        const unsigned left = own.shifted(-1);
#pragma unroll
        for (int d = 0; d < ARound<NNB>::ND; d++) {
            const AWord &q = A.q[A.row(d)];
            for (unsigned m = own.c & q.shifted(A.dx(d)) & ~(left & q.shifted(A.dx(d) - 1)); m; m &= m - 1) {
                const int x = __ffs(m) - 1;
                const int a = L[arun(Bits, B, want, own, x)], b = L[arun(Bits, B, want, q, x + A.dx(d))];
                if (a != b) uf::unite(L, a, b);
            }
        }
    }
}

// links to roots (one store, of the final root); roots are counted per box
__global__ void __launch_bounds__(256) k_al_flatten(ABox *boxes, const unsigned *__restrict__ wbox, const uint2 *__restrict__ list,
                                                    const unsigned *__restrict__ n, int *L, bool fg) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < *n; i += gridDim.x * blockDim.x) {
        const uint2 e = list[i];
        const int s = (int)e.y, root = uf::find_root(L, s);
        if (root != s) {
            L[s] = root;
        } else {
            ABox &B = boxes[wbox[e.x / 32]];
            atomicAdd(fg ? &B.nfg : &B.nbg, 1u);
        }
    }
}

// f(word index, bits) for the pieces of the run that starts at arena index s in word gw; returns its last local x
template <class F>
__device__ __forceinline__ int run_pieces(const unsigned *__restrict__ Bits, const ABox &B, unsigned want, unsigned gw, int s, F f) {
    const WordAt a = word_at(B, gw - B.bw0);
    int w = a.w;
    const int b = s - (int)(B.arena + (long long)a.lr * B.n[0]) - 32 * w;
    unsigned piece = piece_at(ab_class(Bits, B, a.lr, (unsigned)w, want), b);
    for (;;) {
        f(B.bw0 + a.lr * B.W + (unsigned)w, piece);
        if (!(piece >> 31) || w + 1 >= (int)B.W) break;
        const unsigned c = ab_class(Bits, B, a.lr, (unsigned)w + 1u, want);
        if (!(c & 1u)) break;
        piece = piece_at(c, 0);
        w++;
    }
    return 32 * w + 31 - __clz(piece);
}

// background components touching a face of the box flag their root
__global__ void __launch_bounds__(256) k_al_edges(const ABox *boxes, const unsigned *__restrict__ wbox,
                                                  const unsigned *__restrict__ Bits, const uint2 *__restrict__ list,
                                                  const unsigned *__restrict__ n, const int *L, unsigned char *edge) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < *n; i += gridDim.x * blockDim.x) {
        const uint2 e = list[i];
        const ABox &B = boxes[wbox[e.x / 32]];
        const WordAt a = word_at(B, e.x - B.bw0);
        const int n1 = B.n[1], z = (int)(a.lr / (unsigned)n1), y = (int)(a.lr - (unsigned)z * (unsigned)n1);
        const bool face = y == 0 || z == 0 || y == n1 - 1 || z == B.n[2] - 1 || (int)e.y == (int)(B.arena + (long long)a.lr * B.n[0]);
        if (!face && run_pieces(Bits, B, 0u, e.x, (int)e.y, [](unsigned, unsigned) {}) < B.n[0] - 1) continue;
        const int r = L[e.y];
        if (!edge[r]) edge[r] = 1;
    }
}

// bubbles (background components away from the box faces) become foreground,
// when the box's background has at least two components (src/bwlabel.c:488-491)
__global__ void __launch_bounds__(256) k_al_fill(const ABox *boxes, const unsigned *__restrict__ wbox,
                                                 const unsigned *__restrict__ Bits, const uint2 *__restrict__ list,
                                                 const unsigned *__restrict__ n, const int *L, const unsigned char *__restrict__ edge,
                                                 unsigned *out) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < *n; i += gridDim.x * blockDim.x) {
        const uint2 e = list[i];
        const ABox &B = boxes[wbox[e.x / 32]];
        if (B.nbg < 2 || edge[L[e.y]]) continue;
        run_pieces(Bits, B, 0u, e.x, (int)e.y, [&](unsigned w, unsigned piece) { atomicOr(out + w, piece); });
    }
}

// component sizes at the roots; lanes whose root is the first one's add up first
__global__ void __launch_bounds__(256) k_al_sizes(const ABox *boxes, const unsigned *__restrict__ wbox,
                                                  const unsigned *__restrict__ Bits, const uint2 *__restrict__ list,
                                                  const unsigned *__restrict__ n, const int *L, unsigned *cnt) {
    grid_wait();
    const unsigned n32 = (*n + 31u) & ~31u;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n32; i += gridDim.x * blockDim.x) {   // whole warps
        int root = -1;
        unsigned len = 0;
        if (i < *n) {
            const uint2 e = list[i];
            root = L[e.y];
            run_pieces(Bits, boxes[wbox[e.x / 32]], 1u, e.x, (int)e.y, [&](unsigned, unsigned piece) { len += __popc(piece); });
        }
        const int r0 = __shfl_sync(FULL, root, 0);   // the first lane always has a run
        const unsigned sum = __reduce_add_sync(FULL, root == r0 ? len : 0u);
        if ((threadIdx.x & 31) == 0) atomicAdd(&cnt[r0], sum);
        else if (root >= 0 && root != r0) atomicAdd(&cnt[root], len);
    }
}

// largest component per box; ties go to the smallest root (first in raster order)
__global__ void __launch_bounds__(256) k_al_best(ABox *boxes, const unsigned *__restrict__ wbox, const uint2 *__restrict__ list,
                                                 const unsigned *__restrict__ n, const int *L, const unsigned *__restrict__ cnt) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < *n; i += gridDim.x * blockDim.x) {
        const uint2 e = list[i];
        const int s = (int)e.y;
        if (L[s] != s) continue;
        ABox &B = boxes[wbox[e.x / 32]];
        atomicMax(&B.best, ((unsigned long long)cnt[s] << 32) | (0xffffffffu - (unsigned)(s - B.arena)));
    }
}

// bits of the voxels of each box's largest component (K cleared before)
__global__ void __launch_bounds__(256) k_al_keep(const ABox *boxes, const unsigned *__restrict__ wbox,
                                                 const unsigned *__restrict__ Bits, const uint2 *__restrict__ list,
                                                 const unsigned *__restrict__ n, const int *L, unsigned *K) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < *n; i += gridDim.x * blockDim.x) {
        const uint2 e = list[i];
        const ABox &B = boxes[wbox[e.x / 32]];
        if (!B.best || (long long)L[e.y] != B.arena + (long long)(0xffffffffu - (unsigned)(B.best & 0xffffffffu))) continue;
        run_pieces(Bits, B, 1u, e.x, (int)e.y, [&](unsigned w, unsigned piece) { atomicOr(K + w, piece); });
    }
}

// What the clustering does to the values of a sub-box, applied where they are read
// (agval): kept voxels (K) raised to the box's isolevel when FILL; with LARGEST, a voxel
// neither kept nor, away from the volume faces, next to a kept voxel (all 26 neighbours
// except (-1,-1,-1), src/meshify.c:252) becomes the box minimum (src/meshify.c:332-342).
struct APost {
    const unsigned *K, *KD;   // kept voxels; with LARGEST, those and their neighbours
    const unsigned *S;        // sign of value - iso
    bool fill, largest;
};

// ---- S4: signs and bbox of the clustered sub-boxes -------------------------------------
// A lane per word.  Only the voxels whose value the bits do not settle are read (those next to
// kept ones): 23 M arena voxels took 249 us to write clustered and 67 us to read back,
// 62 us this way.  A sub-box that is the whole volume has every value read for its
// minimum; any other one reaches 0, the smallest possible.
__global__ void __launch_bounds__(256) k_ab_shell(ABox *boxes, const unsigned *__restrict__ wbox, unsigned nbw, APost P, unsigned *S, unsigned *KD,
                                                  const float *__restrict__ arena, int nx, int ny, int nz) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    // rows used: 0..2 = y-1..y+1 in slice z, 3..5 in slice z+1, 6 = (y, z-1), 7 = (y+1, z-1), 8 = (y-1, z-1)
    constexpr int DY[9] = {-1, 0, 1, -1, 0, 1, 0, 1, -1}, DZ[9] = {0, 0, 0, 1, 1, 1, -1, -1, -1};
    for (unsigned w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; w0 < nbw; w0 += gridDim.x * blockDim.x) {
        ABox &B = boxes[wbox[w0 / 32]];
        const WordAt a = word_at(B, w0 - B.bw0 + (unsigned)lane);
        const int n1 = B.n[1], n2 = B.n[2], z = (int)(a.lr / (unsigned)n1), y = (int)(a.lr - (unsigned)z * (unsigned)n1);
        const unsigned valid = a.live ? ab_valid(B, (unsigned)a.w) : 0u, W = B.W;
        unsigned on = 0u, kept = 0u;
        if (P.K) {
#pragma unroll
            for (int k = 0; k < 9; k++) {
                if (!P.largest && k != 1) continue;
                const int yy = y + DY[k], zz = z + DZ[k];
                const bool in = a.live && yy >= 0 && zz >= 0 && yy < n1 && zz < n2;
                const unsigned q = in ? B.bw0 + ((unsigned)zz * (unsigned)n1 + (unsigned)yy) * W + (unsigned)a.w : 0u;
                const unsigned cur = in ? __ldg(P.K + q) : 0u;
                unsigned prv = __shfl_up_sync(FULL, cur, 1), nxt = __shfl_down_sync(FULL, cur, 1);
                if (lane == 0) prv = in && a.w ? __ldg(P.K + q - 1) : 0u;
                if (lane == 31) nxt = in && a.w + 1 < (int)W ? __ldg(P.K + q + 1) : 0u;
                if (a.w == 0) prv = 0u;
                if (a.w + 1 >= (int)W) nxt = 0u;
                on |= cur | (cur >> 1) | (nxt << 31) | (k < 8 ? (cur << 1) | (prv >> 31) : 0u);   // row 8: no K(x-1)
                if (k == 1) kept = cur;
            }
        }
        unsigned shell = valid & ~kept, masked = 0u;
        if (P.largest) {
            const int gy = B.o[1] + y, gz = B.o[2] + z, gx0 = B.o[0] + 32 * a.w;
            if (gy > 0 && gz > 0 && gy < ny - 1 && gz < nz - 1) on &= mcw::bit_range(1 - gx0, nx - 1 - gx0);
            else on = 0u;
            shell &= on;
            masked = valid & ~(kept | shell);
        }
        const float iso = B.iso, vmin = ord2f(B.vmin);
        const unsigned vsig = __fsub_rn(vmin, iso) > -N2M_FLT_EPS ? FULL : 0u, vge = vmin >= iso ? FULL : 0u;
        unsigned sg = kept | (masked & vsig), ge = kept | (masked & vge);
        const unsigned read = B.full ? valid & ~masked : shell;
        float lo = INFINITY;
        if (B.full && masked) lo = vmin;
        const float *base = arena + B.arena;
        for (unsigned busy = __ballot_sync(FULL, read != 0u); busy;) {   // four words in flight
            int j[4];
            float val[4];
            unsigned rj[4], kj[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                j[u] = busy ? __ffs(busy) - 1 : -1;
                busy &= busy - 1u;
                rj[u] = __shfl_sync(FULL, read, j[u] & 31);
                kj[u] = __shfl_sync(FULL, kept, j[u] & 31);
                const unsigned lr = __shfl_sync(FULL, a.lr, j[u] & 31);
                const int w = __shfl_sync(FULL, a.w, j[u] & 31);
                val[u] = j[u] >= 0 && (rj[u] >> lane & 1u) ? __ldg(base + (long long)lr * B.n[0] + 32 * w + lane) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const bool in = j[u] >= 0 && (rj[u] >> lane & 1u), k = kj[u] >> lane & 1u;
                if (in) lo = fminf(lo, k && P.fill ? fmaxf(val[u], iso) : val[u]);
                const unsigned g = __ballot_sync(FULL, in && !k && val[u] >= iso),
                               p = __ballot_sync(FULL, in && !k && __fsub_rn(val[u], iso) > -N2M_FLT_EPS);
                if (lane == j[u]) {
                    ge |= g;
                    sg |= p;
                }
            }
        }
        S[w0 + (unsigned)lane] = sg;   // the filling too
        if (P.largest) KD[w0 + (unsigned)lane] = kept | shell;
        if (B.full) {
            for (int o = 16; o; o >>= 1) lo = fminf(lo, __shfl_xor_sync(FULL, lo, o));
            if (lane == 0 && lo < INFINITY) atomicMin(&B.amin, f2ord(lo));
        }
        if (__any_sync(FULL, ge != 0u)) {
            int x0 = ge ? 32 * a.w + __ffs(ge) - 1 : INT_MAX, x1 = ge ? 32 * a.w + 31 - __clz(ge) : INT_MIN;
            int e[6] = {__reduce_min_sync(FULL, x0), __reduce_min_sync(FULL, ge ? y : INT_MAX), __reduce_min_sync(FULL, ge ? z : INT_MAX),
                        __reduce_max_sync(FULL, x1), __reduce_max_sync(FULL, ge ? y : INT_MIN), __reduce_max_sync(FULL, ge ? z : INT_MIN)};
            if (lane == 0) {
                for (int k = 0; k < 3; k++) {
                    const int l = B.o[k] + e[k], h = B.o[k] + e[k + 3];
                    if (l < *(volatile int *)&B.blo[k]) atomicMin(&B.blo[k], l);
                    if (h > *(volatile int *)&B.bhi[k]) atomicMax(&B.bhi[k], h);
                }
            }
        }
    }
}

__global__ void k_a_pad(ABox *boxes, int nb) {
    grid_wait();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    ABox &B = boxes[b];
    float amin = ord2f(B.amin);
    if (!B.full) amin = fminf(amin, 0.f);
    B.pad = __fsub_rn(fminf(amin, B.edge_max), B.iso);
}

// ---- S5-S7: marching cubes over every label's padded grid ------------------------------
// grid value (x,y,z) of box B minus isolevel, as the single-volume gval
__device__ __forceinline__ float agval(const AtlasVol &v, const ABox &B, const APost &P, const float *arena, int x, int y, int z) {
    const long long j = (long long)(B.glo[0] + x) + (long long)(y + B.glo[1]) * v.nx + (long long)(z + B.glo[2]) * v.nxy;
    float val;
    if (j < v.nvox) {
        // the box grid ends at the volume's dims: a coordinate past them by one wraps into the next row / slice
        int vx = B.glo[0] + x, vy = y + B.glo[1], vz = z + B.glo[2];
        if (vx >= v.nx) {
            vx -= v.nx;
            vy++;
        }
        if (vy >= v.ny) {
            vy -= v.ny;
            vz++;
        }
        const int lx = vx - B.o[0], ly = vy - B.o[1], lz = vz - B.o[2];
        val = 0.f;
        if (lx >= 0 && ly >= 0 && lz >= 0 && lx < B.n[0] && ly < B.n[1] && lz < B.n[2]) {
            const unsigned lr = (unsigned)lz * (unsigned)B.n[1] + (unsigned)ly, w = B.bw0 + lr * B.W + ((unsigned)lx >> 5);
            val = __ldg(arena + B.arena + (long long)lr * B.n[0] + lx);
            if (P.largest && !(__ldg(P.KD + w) >> (lx & 31) & 1u)) val = ord2f(B.vmin);
            else if (P.fill && (__ldg(P.K + w) >> (lx & 31) & 1u)) val = fmaxf(val, B.iso);
        }
        if (vx == 0 || vy == 0 || vz == 0 || vx == v.nx - 1 || vy == v.ny - 1 || vz == v.nz - 1)
            val = fminf(B.edge_max, val);
        val = __fsub_rn(val, B.iso);
    } else {
        val = B.pad;
    }
    if (fabsf(val) < N2M_FLT_EPS) val = N2M_FLT_EPS;
    return val;
}

// The grids of all boxes are words of one numbering for mcwords.cuh: each box begins at a
// multiple of SUB words, so that a sub-tile belongs to one box (subbox).
__device__ __forceinline__ unsigned agrid_words(const ABox &B) { return B.WX * (unsigned)B.gn[1] * (unsigned)B.gn[2]; }

// Sign words from the sub-boxes' sign bits, a thread per word and no values read.  A grid
// ends at most one voxel past the volume and two past the sub-box, where values are 0; agval's
// cases by words: darkening is min(edge_max, value), whose sign is both their signs, a
// coordinate one past the volume wraps into the next row or slice (whose first
// voxels are on a face), and past the last one there is padding.
__global__ void __launch_bounds__(256) k_a_signs(AtlasVol v, const ABox *boxes, int nb, unsigned nsub, const unsigned *__restrict__ S,
                                                 unsigned *signs, unsigned *subbox) {
    grid_wait();
    const unsigned lane = threadIdx.x & 31u;
    for (unsigned sub = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; sub < nsub; sub += (gridDim.x * blockDim.x) >> 5) {
        const int b = find_item(boxes, nb, sub * mcw::SUB, &ABox::word0);
        const ABox &B = boxes[b];
        if (lane == 0) subbox[sub] = (unsigned)b;
        const unsigned lw = sub * mcw::SUB - B.word0 + lane;
        unsigned m = 0;
        if (lw < agrid_words(B)) {
            const unsigned row = lw / B.WX;
            const int x0 = 32 * (int)(lw - row * B.WX), z = (int)(row / (unsigned)B.gn[1]), y = (int)(row - (unsigned)z * (unsigned)B.gn[1]);
            const bool dark = __fsub_rn(B.edge_max, B.iso) > -N2M_FLT_EPS, padp = B.pad > -N2M_FLT_EPS;
            const unsigned zero = __fsub_rn(0.f, B.iso) > -N2M_FLT_EPS ? FULL : 0u;
            auto bits = [&](int vx, int vy, int vz) -> unsigned {   // signs of voxels vx .. vx+31 of a row, no face rule
                const int lx = vx - B.o[0], ly = vy - B.o[1], lz = vz - B.o[2];
                if (ly < 0 || lz < 0 || ly >= B.n[1] || lz >= B.n[2] || lx <= -32 || lx >= B.n[0]) return zero;
                const unsigned *r = S + B.bw0 + ((unsigned)lz * (unsigned)B.n[1] + (unsigned)ly) * B.W;
                const unsigned q = (unsigned)(lx < 0 ? 0 : lx) >> 5;
                const unsigned c = __ldg(r + q);
                const unsigned n = lx < 0 ? c << -lx : __funnelshift_r(c, q + 1 < B.W ? __ldg(r + q + 1) : 0u, lx & 31);
                const unsigned in = mcw::bit_range(-lx, B.n[0] - lx);
                return (n & in) | (zero & ~in);
            };
            int vy = B.glo[1] + y, vz = B.glo[2] + z;
            const int vx = B.glo[0] + x0, pad = v.nx - vx;   // bit of the padding column
            const unsigned in = mcw::bit_range(0, B.gn[0] - x0);
            if (vy >= v.ny) {   // the padding row is row 0 of the next slice
                vy -= v.ny;
                vz++;
            }
            if (vz >= v.nz) {
                m = padp ? FULL : 0u;
            } else {
                m = bits(vx, vy, vz);
                if (!dark) {
                    if (vy == 0 || vz == 0 || vy == v.ny - 1 || vz == v.nz - 1) m = 0u;
                    else m &= mcw::bit_range(1 - vx, v.nx - 1 - vx);
                }
                if (pad >= 0 && pad < 32) {
                    m &= mcw::bit_range(0, pad);
                    int py = vy + 1, pz = vz;
                    if (py >= v.ny) {
                        py -= v.ny;
                        pz++;
                    }
                    if (pz < v.nz ? dark && (bits(0, py, pz) & 1u) : padp) m |= 1u << pad;
                }
            }
            m &= in;
        }
        signs[sub * mcw::SUB + lane] = m;
    }
}

// mcwords.cuh's policy for the boxes' padded Lewiner grids.  Vertex numbers are contiguous per
// box: its edge vertices, then its c-vertices.
struct Policy {
    static constexpr bool MULTI = true, REVERSE = true, CVERTS = true;
    static constexpr int CTAS = 8, EV = 1;
    AtlasVol v;
    const ABox *boxes;
    int nb;
    const unsigned *subbox;
    APost post;
    const float *arena;
    bool classic;
    vec3d *pts;
    int *cand, *ccand;
    unsigned *ncand, *nccand;
    int cap;
    unsigned *near;
    __device__ __forceinline__ unsigned quick(int lut) const {
        Tiling T = {0, 0, false};
        return quick_tiling(lut, classic, T) ? (unsigned)T.off << 8 | (unsigned)T.n : mcw::TESTS;
    }
    __device__ __forceinline__ int code(int off) const { return d_lut[off]; }
    __device__ __forceinline__ bool geo(unsigned w, mcw::Geo &q) const {
        const unsigned b = __ldg(subbox + w / mcw::SUB);
        const ABox &B = boxes[b];
        const unsigned lw = w - B.word0, row = lw / B.WX, xw = lw - row * B.WX;
        q.z = (int)(row / (unsigned)B.gn[1]);
        if (q.z >= B.gn[2]) return false;   // the filling behind the box's last word
        q.y = (int)(row - (unsigned)q.z * (unsigned)B.gn[1]);
        q.x0 = 32 * (int)xw;
        q.WX = B.WX;
        q.slice = B.WX * (unsigned)B.gn[1];
        q.inm = mcw::bit_range(0, B.gn[0] - q.x0);
        q.hxm = mcw::bit_range(0, B.gn[0] - 1 - q.x0);
        q.hy = q.y < B.gn[1] - 1;
        q.hz = q.z < B.gn[2] - 1;
        q.nx = xw + 1 < B.WX;
        q.tag = (int)b;
        return true;
    }
    __device__ __forceinline__ void voxel_word(const mcw::Geo &, int &wx, int &vy, int &vz) const { wx = vy = vz = 0; }
    __device__ __forceinline__ void shifts(const mcw::Out &o, unsigned s, const uint4 &total, unsigned &e, unsigned &c) const {
        const ABox &B = boxes[__ldg(subbox + s)];
        const unsigned s0 = B.word0 / mcw::SUB, s1 = s0 + (agrid_words(B) + mcw::SUB - 1) / mcw::SUB;
        e = mcw::sub_offset(o, s0).z;                             // earlier boxes' c-vertices
        c = s1 < o.nsub ? mcw::sub_offset(o, s1).x : total.x;     // edge vertices up to the end of this box
    }
    __device__ __forceinline__ void corners(const ABox &B, int x, int y, int z, float *c) const {
        c[0] = agval(v, B, post, arena, x, y, z); c[1] = agval(v, B, post, arena, x + 1, y, z);
        c[2] = agval(v, B, post, arena, x + 1, y + 1, z); c[3] = agval(v, B, post, arena, x, y + 1, z);
        c[4] = agval(v, B, post, arena, x, y, z + 1); c[5] = agval(v, B, post, arena, x + 1, y, z + 1);
        c[6] = agval(v, B, post, arena, x + 1, y + 1, z + 1); c[7] = agval(v, B, post, arena, x, y + 1, z + 1);
    }
    __device__ __noinline__ mcw::CubeTiling tests(const mcw::Geo &q, int x, int y, int z, int lut) const {
        float c[8];
        corners(boxes[q.tag], x, y, z, c);
        const Tiling T = select_tiling(c, lut, classic);
        return mcw::CubeTiling{T.off, T.n, T.cv};
    }
    __device__ __forceinline__ void cvertex(const mcw::Geo &q, int x, int y, int z, int id) const {
        const ABox &B = boxes[q.tag];
        float c[8];
        corners(B, x, y, z, c);
        emit_cvertex(c, x, y, z, (float)B.glo[0], (float)B.glo[1], (float)B.glo[2], id, pts, ccand, nccand, cap);
        mark_near(near, id);
    }
    struct Edge {
        float c0, c1, flo0, flo1, flo2;
    };
    __device__ __forceinline__ Edge edge(int x, int y, int z, int ax, int tag) const {
        const ABox &B = boxes[tag];
        return Edge{agval(v, B, post, arena, x, y, z), agval(v, B, post, arena, x + (ax == 0), y + (ax == 1), z + (ax == 2)),
                    (float)B.glo[0], (float)B.glo[1], (float)B.glo[2]};
    }
    __device__ __forceinline__ vec3d vertex(const Edge &c, int x, int y, int z, int ax, int id) const {
        return edge_vertex(c.c0, c.c1, x, y, z, ax, c.flo0, c.flo1, c.flo2, id, cand, ncand, cap, near);
    }
};

// per box: edge vertices, triangles and c-vertices of all earlier boxes, from which its
// contiguous ranges follow (and the totals after the last)
struct BoxOff {
    unsigned e, t, c;
};
__global__ void k_a_boxoff(const ABox *boxes, int nb, mcw::Out o, BoxOff *boff) {
    grid_wait();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nb) return;
    const unsigned s = b < nb ? boxes[b].word0 / mcw::SUB : o.nsub;
    const uint4 q = s < o.nsub ? mcw::sub_offset(o, s) : *o.total;
    boff[b] = {q.x, q.y, q.z};
}

// binarise the whole volume for one label (the per-label loop)
__global__ void k_binarize(const short *lab, long long n, int label, float *out) {
    grid_wait();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = lab[i] == label ? 1.f : 0.f;
}

__global__ void k_offset_tris(vec3i *t, int n, int off) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        t[i].x -= off; t[i].y -= off; t[i].z -= off;
    }
}
}  // namespace


// ---- host side ------------------------------------------------------------------------
namespace {
inline unsigned pgrid(unsigned items, unsigned per_sm) {
    const unsigned cap = 152u * per_sm;
    return std::max(1u, std::min(items, cap));
}

double d3(const vec3d &a, const vec3d &b) {
    const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
    return sqrt(dx * dx + dy * dy + dz * dz);
}
uint32_t kbits(float f) {
    uint32_t u;
    memcpy(&u, &f, 4);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__global__ void k_a_fill_bb(int *bb, int n) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) bb[i] = (i % 6) < 3 ? INT_MAX : INT_MIN;
}

__global__ void k_a_gather(const vec3d *p, const int *ids, int n, vec3d *out) {
    grid_wait();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = p[ids[i]];
}

// kept triangles before each box's first triangle, from the degenerate filter's bits
__global__ void k_a_kept(const unsigned *tri_start, int nb, unsigned nt, const unsigned *bits, const unsigned *tile_off,
                         const unsigned *total_kept, unsigned *kept_before) {
    grid_wait();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b > nb) return;
    const unsigned t = tri_start[b];
    unsigned k;
    if (t >= nt) k = *total_kept;
    else {
        k = tile_off[t / DEG_TILE];
        for (unsigned w = t / DEG_TILE * (DEG_TILE / 32); w < t / 32; w++) k += __popc(bits[w]);
        k += __popc(bits[t / 32] & ((1u << (t & 31u)) - 1u));
    }
    kept_before[b] = k;
}

// triangle indices relative to their own mesh
__global__ void k_a_localize(vec3i *t, unsigned nt, const unsigned *tri_start, const unsigned *vert_start, int nb) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
        int lo = 0, hi = nb - 1;
        while (lo < hi) {
            const int m = (lo + hi + 1) >> 1;
            if (tri_start[m] <= i) lo = m;
            else hi = m - 1;
        }
        const int o = (int)vert_start[lo];
        t[i].x -= o; t[i].y -= o; t[i].z -= o;
    }
}
}  // namespace

namespace {
// smoothing, isolevel, clustering and signs/bbox: device-only work (no host
// synchronisation)
struct Segment {
    AtlasVol v;
    ABox *db;
    int nb;
    unsigned tiles;
    float *ar;
    bool smooth_on, only_largest, fill_bubbles;
    int nx, ny, nz;
    long long arena;
    unsigned nrows, nbw;   // rows and bit words of all the boxes
    APost post;            // what the clustering leaves (enqueue)

    n2m_status ensure(AtlasWork &w) {
        CKS(w.keep.ensure((size_t)nbw * sizeof(unsigned)));
        CKS(w.shell.ensure((size_t)2 * nbw * sizeof(unsigned)));
        CKS(w.wbox.ensure((size_t)nbw / 32 * sizeof(unsigned)));
        if (only_largest || fill_bubbles) {
            CKS(w.mask.ensure((size_t)nbw * sizeof(unsigned)));
            CKS(w.lab.ensure((size_t)arena * sizeof(int)));
            CKS(w.list.ensure(((size_t)arena + nrows) / 2 * sizeof(uint2)));   // every second voxel of a row at most
            CKS(w.wlist.ensure(((size_t)nbw + 4) * sizeof(unsigned)));
            if (fill_bubbles) CKS(w.fill.ensure((size_t)nbw * sizeof(unsigned)));
            if (fill_bubbles) CKS(w.edge.ensure((size_t)arena));
            if (only_largest) CKS(w.ucnt.ensure((size_t)arena * sizeof(unsigned)));
        }
        return N2M_OK;
    }

    n2m_status enqueue(AtlasWork &w, cudaStream_t s) {
        unsigned *wbox = w.wbox.as<unsigned>();
        unsigned *M = w.keep.as<unsigned>();   // the labels' masks, until the kept voxels take their place
        const unsigned wg = std::max(1u, std::min((nbw + 255) / 256, 152u * 16u));   // a thread per word
        n2m_launch(k_a_mask, wg, 256, 0, s, v, db, nb, nbw, M, wbox);
        n2m_launch(k_a_smooth, std::max(1u, std::min((tiles + AWARPS - 1) / AWARPS, 152u * 8u)), 32 * AWARPS, 0, s, db, nb, tiles,
                   M, ar, nx, ny, nz, smooth_on);
        n2m_launch(k_a_iso, (nb + 127) / 128, 128, 0, s, db, nb);
        if (only_largest || fill_bubbles) {
            unsigned *Bm = w.mask.as<unsigned>();
            int *L = w.lab.as<int>();
            // lists by words, then a thread per entry (about one run per word)
            const unsigned lg = std::max(1u, std::min((nbw + 256 * AL_K - 1) / (256 * AL_K), 152u * 16u)), g = std::min(wg, 152u * 8u);
            uint2 *list = w.list.as<uint2>();
            unsigned *wlist = w.wlist.as<unsigned>(), *n = wlist + nbw;   // {runs, words} of the background, of the foreground
            CK(cudaMemsetAsync(n, 0, 4 * sizeof(unsigned), s));
            n2m_launch(k_ab_bits, wg, 256, 0, s, db, wbox, nbw, ar, Bm);
            const unsigned *K = Bm;
            if (fill_bubbles) {
                unsigned char *edge = w.edge.as<unsigned char>();
                unsigned *Fm = w.fill.as<unsigned>();
                n2m_launch(k_al_list<3>, lg, 256, 0, s, db, wbox, nbw, Bm, 0u, list, wlist, n, L, edge, nullptr);
                n2m_launch(k_al_jump, g, 256, 0, s, list, n, L);
                n2m_launch(k_al_merge<3>, g, 256, 0, s, db, wbox, Bm, 0u, wlist, n, L);
                n2m_launch(k_al_flatten, g, 256, 0, s, db, wbox, list, n, L, false);
                n2m_launch(k_al_edges, g, 256, 0, s, db, wbox, Bm, list, n, L, edge);
                CK(cudaMemcpyAsync(Fm, Bm, (size_t)nbw * sizeof(unsigned), cudaMemcpyDeviceToDevice, s));
                n2m_launch(k_al_fill, g, 256, 0, s, db, wbox, Bm, list, n, L, edge, Fm);
                K = Fm;
            }
            if (only_largest) {
                const unsigned *F = K;   // the (filled) foreground
                unsigned *cnt = w.ucnt.as<unsigned>(), *Kb = w.keep.as<unsigned>();
                n2m_launch(k_al_list<9>, lg, 256, 0, s, db, wbox, nbw, F, 1u, list, wlist, n + 2, L, nullptr, cnt);
                n2m_launch(k_al_jump, g, 256, 0, s, list, n + 2, L);
                n2m_launch(k_al_merge<9>, g, 256, 0, s, db, wbox, F, 1u, wlist, n + 2, L);
                n2m_launch(k_al_flatten, g, 256, 0, s, db, wbox, list, n + 2, L, true);
                n2m_launch(k_al_sizes, g, 256, 0, s, db, wbox, F, list, n + 2, L, cnt);
                n2m_launch(k_al_best, g, 256, 0, s, db, wbox, list, n + 2, L, cnt);
                CK(cudaMemsetAsync(Kb, 0, (size_t)nbw * sizeof(unsigned), s));
                n2m_launch(k_al_keep, g, 256, 0, s, db, wbox, F, list, n + 2, L, Kb);
                K = Kb;
            }
            post.K = K;
        }
        post.fill = fill_bubbles;
        post.largest = only_largest;
        unsigned *S = w.shell.as<unsigned>(), *KD = S + nbw;
        post.S = S;
        post.KD = KD;
        n2m_launch(k_ab_shell, wg, 256, 0, s, db, wbox, nbw, post, S, KD, ar, nx, ny, nz);
        n2m_launch(k_a_pad, (nb + 127) / 128, 128, 0, s, db, nb);
        CKL();
        return N2M_OK;
    }
};
}  // namespace

n2m_status atlas_hist(const short *d_lab, const int dim[3], AtlasWork &w, cudaStream_t s, int *maxlab,
                      std::vector<unsigned> &cnt, std::vector<int> &bb) {
    const int ML = 32767;
    CKS(w.cnt.ensure((ML + 1) * sizeof(unsigned)));
    CKS(w.bb.ensure((size_t)(ML + 1) * 6 * sizeof(int) + 16));
    CK(cudaMemsetAsync(w.cnt.p, 0, (ML + 1) * sizeof(unsigned), s));
    int *dvmax = (int *)(w.bb.as<int>() + (ML + 1) * 6);
    CK(cudaMemsetAsync(dvmax, 0, sizeof(int), s));
    n2m_launch(k_a_fill_bb, 256, 256, 0, s, w.bb.as<int>(), (ML + 1) * 6);
    AtlasVol v{d_lab, dim[0], dim[1], dim[2], (long long)dim[0] * dim[1], (long long)dim[0] * dim[1] * dim[2]};
    n2m_launch(k_a_hist, pgrid((unsigned)std::min<long long>((v.nvox + 256 * HV - 1) / (256 * HV), 1u << 30), 4), HT, 0, s, v, ML,
               w.cnt.as<unsigned>(), w.bb.as<int>(), dvmax);
    CKL();
    int mx = 0;
    CK(cudaMemcpyAsync(&mx, dvmax, sizeof(int), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    *maxlab = mx;
    cnt.assign(mx + 1, 0u);
    bb.assign((size_t)(mx + 1) * 6, 0);
    if (mx >= 1) {
        CK(cudaMemcpyAsync(cnt.data(), w.cnt.p, (mx + 1) * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        CK(cudaMemcpyAsync(bb.data(), w.bb.p, (size_t)(mx + 1) * 6 * sizeof(int), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
    }
    return N2M_OK;
}

n2m_status atlas_binarize(const short *d_lab, long long n, int label, float *out, cudaStream_t s) {
    n2m_launch(k_binarize, pgrid((unsigned)std::min<long long>((n + 255) / 256, 1u << 30), 32), 256, 0, s, d_lab, n, label,
               out);
    CKL();
    return N2M_OK;
}

n2m_status atlas_offset_tris(vec3i *t, int n, int off, cudaStream_t s) {
    if (n > 0 && off) n2m_launch(k_offset_tris, pgrid((n + 255) / 256, 16), 256, 0, s, t, n, off);
    CKL();
    return N2M_OK;
}

n2m_status atlas_batched(const short *d_lab, const int dim[3], const n2m_options &o, AtlasWork &w, ScanWork &sw,
                         DegWork &dw, HcWork &hw, cudaStream_t s, std::vector<n2m_atlas_mesh> &out, vec3d **d_pts,
                         vec3i **d_tris, int64_t *npts, int64_t *ntris, float *ms_stage) {
    cudaEvent_t ev[6];
    for (auto &e : ev) CK(cudaEventCreate(&e));
    struct EvGuard {
        cudaEvent_t *e;
        ~EvGuard() { for (int i = 0; i < 6; i++) cudaEventDestroy(e[i]); }
    } guard{ev};
    CK(cudaEventRecord(ev[0], s));
    int maxlab = 0;
    std::vector<unsigned> cnt;
    std::vector<int> bb;
    CKS(atlas_hist(d_lab, dim, w, s, &maxlab, cnt, bb));
    if (maxlab < 1) {
        n2m_set_error("intensity range not consistent with an indexed atlas");
        return N2M_ERR_BAD_ARGS;
    }
    AtlasVol v{d_lab, dim[0], dim[1], dim[2], (long long)dim[0] * dim[1], (long long)dim[0] * dim[1] * dim[2]};
    // ---- sub-boxes
    std::vector<ABox> boxes;
    long long arena = 0;
    unsigned tiles = 0;
    unsigned long long rows = 0, bwords = 0;
    for (int l = 1; l <= maxlab; l++) {
        if (!cnt[l]) continue;
        ABox B;
        memset(&B, 0, sizeof(B));
        B.label = l;
        bool full = true;
        for (int a = 0; a < 3; a++) {
            const int lo = std::max(bb[6 * l + a] - 3, 0), hi = std::min(bb[6 * l + 3 + a] + 3, dim[a] - 1);
            B.o[a] = lo;
            B.n[a] = hi - lo + 1;
            full = full && lo == 0 && B.n[a] == dim[a];
        }
        B.full = full;
        B.arena = arena;
        arena += (long long)B.n[0] * B.n[1] * B.n[2];
        B.tile0 = tiles;
        B.W = (unsigned)(B.n[0] + 31) / 32;
        tiles += B.W * (unsigned)((B.n[1] + ARY - 1) / ARY) * (unsigned)((B.n[2] + AZC - 1) / AZC);
        B.bw0 = bwords;
        rows += (unsigned long long)B.n[1] * B.n[2];
        bwords += ((unsigned long long)B.W * B.n[1] * B.n[2] + 31) / 32 * 32;
        B.vmin = INT_MAX;
        B.vmax = INT_MIN;
        for (int a = 0; a < 3; a++) { B.blo[a] = INT_MAX; B.bhi[a] = INT_MIN; }
        boxes.push_back(B);
    }
    const int nb = (int)boxes.size();
    if (arena >= 0x7fffffffLL) {
        n2m_set_error("atlas arena exceeds 2^31 voxels");
        return N2M_ERR_TOO_LARGE;
    }
    CKS(w.boxes.ensure((size_t)nb * sizeof(ABox)));
    CKS(w.arena.ensure((size_t)arena * sizeof(float)));
    ABox *db = w.boxes.as<ABox>();
    CK(cudaMemcpyAsync(db, boxes.data(), nb * sizeof(ABox), cudaMemcpyHostToDevice, s));
    float *ar = w.arena.as<float>();
    const bool smooth_on = o.pre_smooth && dim[0] >= 5 && dim[1] >= 5 && dim[2] >= 5;
    Segment seg{v, db, nb, tiles, ar, smooth_on, o.only_largest, o.fill_bubbles, dim[0], dim[1], dim[2], arena,
                (unsigned)rows, (unsigned)bwords, APost{}};
    CKS(seg.ensure(w));
    CK(cudaEventRecord(ev[1], s));
    CKS(seg.enqueue(w, s));
    CK(cudaEventRecord(ev[2], s));
    CK(cudaMemcpyAsync(boxes.data(), db, nb * sizeof(ABox), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    CK(cudaEventRecord(ev[3], s));
    // ---- marching-cubes grids
    unsigned long long words64 = 0;
    for (auto &B : boxes) {
        if (!B.fail && B.blo[0] > B.bhi[0]) B.fail = N2M_ERR_EMPTY;
        B.word0 = (unsigned)words64;
        if (B.fail) {
            B.WX = 0;
            for (int a = 0; a < 3; a++) B.gn[a] = 0;
            continue;
        }
        for (int a = 0; a < 3; a++) {
            const int lo = std::max(B.blo[a] - 1, 0), hi = std::min(B.bhi[a] + 2, dim[a]);
            B.glo[a] = lo;
            B.gn[a] = hi - lo + 1;
        }
        B.WX = (unsigned)((B.gn[0] + 31) / 32);
        words64 += ((unsigned long long)B.WX * (unsigned)B.gn[1] * (unsigned)B.gn[2] + mcw::SUB - 1) / mcw::SUB * mcw::SUB;
    }
    if (words64 >= 0xffffffffULL - mcw::SUB) {
        n2m_set_error("atlas grids too large");
        return N2M_ERR_TOO_LARGE;
    }
    const unsigned words = (unsigned)words64, nsub = words / mcw::SUB;
    CK(cudaMemcpyAsync(db, boxes.data(), nb * sizeof(ABox), cudaMemcpyHostToDevice, s));
    CKS(w.tot.ensure(sizeof(MarchOut) + (size_t)(nb + 1) * sizeof(BoxOff)));
    MarchOut *dm = w.tot.as<MarchOut>();
    BoxOff *dboff = (BoxOff *)(dm + 1);
    const bool classic = o.cubes == N2M_CUBES_CLASSIC_TABLE;
    std::vector<BoxOff> boff(nb + 1, BoxOff{0u, 0u, 0u});
    mcw::Out mo{};
    Policy pol{v, db, nb, nullptr, seg.post, ar, classic, nullptr, nullptr, nullptr, &dm->ncand, &dm->nccand, 0, nullptr};
    CK(cudaMemsetAsync(dm, 0, sizeof(uint4) + 4 * sizeof(unsigned), s));
    if (words) {
        CKS(mcw::prepare(w.mc, words, &dm->tot, mo));
        CKS(w.mc.signs.ensure((size_t)words * sizeof(unsigned)));
        CKS(w.subbox.ensure((size_t)nsub * sizeof(unsigned)));
        unsigned *signs = w.mc.signs.as<unsigned>();
        pol.subbox = w.subbox.as<unsigned>();
        n2m_launch(k_a_signs, std::max(1u, std::min((nsub + 7) / 8, 152u * 16u)), 256, 0, s, v, db, nb, nsub, seg.post.S, signs,
                   w.subbox.as<unsigned>());
        CKS(mcw::count_signs(pol, signs, mo, mcw::Marks{nullptr, 0, 0, 0, 0}, s));
        CKS(mcw::count_values(pol, signs, w.mc, mo, !classic, s));
        n2m_launch(k_a_boxoff, (nb + 128) / 128, 128, 0, s, db, nb, mo, dboff);
        CKL();
        CK(cudaMemcpyAsync(boff.data(), dboff, (nb + 1) * sizeof(BoxOff), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
    }
    const unsigned nv = boff[nb].e + boff[nb].c, nt = boff[nb].t;
    CKS(w.pts.ensure((size_t)std::max(nv, 1u) * sizeof(vec3d)));
    CKS(w.tris.ensure((size_t)std::max(nt, 1u) * sizeof(vec3i)));
    const int cap = (int)std::min<unsigned>(nv / 16 + 65536, 1u << 26);
    CKS(w.cand.ensure((size_t)2 * cap * sizeof(int)));
    int *cand = w.cand.as<int>();
    unsigned *ncand = &dm->ncand, *near = nullptr;
    if (std::max({dim[0], dim[1], dim[2]}) < 1 << 22) {   // NEAR_CORNER
        CKS(dw.near.ensure(((size_t)nv + 31) / 32 * sizeof(unsigned)));
        near = dw.near.as<unsigned>();
        CK(cudaMemsetAsync(near, 0, ((size_t)nv + 31) / 32 * sizeof(unsigned), s));
    }
    if (nv || nt) {
        pol.pts = w.pts.as<vec3d>();
        pol.cand = cand;
        pol.ccand = cand + cap;
        pol.cap = cap;
        pol.near = near;
        CKS(mcw::emit(pol, w.mc.signs.as<unsigned>(), w.mc, mo, MeshRoom{nv, nt}, w.tris.as<vec3i>(), s));
    }
    unsigned nc[2];
    CK(cudaMemcpyAsync(nc, ncand, 2 * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    CK(cudaEventRecord(ev[4], s));
    if (nc[0] > (unsigned)cap || nc[1] > (unsigned)cap) {
        n2m_set_error("weld candidate overflow");
        return N2M_ERR_INTERNAL;
    }
    if (nc[1]) {
        CK(cudaMemcpyAsync(cand + nc[0], cand + cap, nc[1] * sizeof(int), cudaMemcpyDeviceToDevice, s));
        unsigned t2 = nc[0] + nc[1];
        CK(cudaMemcpyAsync(ncand, &t2, sizeof(unsigned), cudaMemcpyHostToDevice, s));
        CKS(mc_ccand_scan(w.pts.as<vec3d>(), (int)nv, cand + cap, (int)nc[1], cand, ncand, cap, s));
        CK(cudaMemcpyAsync(nc, ncand, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
    }
    // per box vertex ranges [vs, ve)
    std::vector<unsigned> vs(nb + 1), ts(nb + 1);
    for (int b = 0; b <= nb; b++) { vs[b] = boff[b].e + boff[b].c; ts[b] = boff[b].t; }
    // ---- weld (per box: the reference welds each label's mesh on its own)
    std::vector<int> removed, keepv, ov_id;
    std::vector<vec3d> ov_pos;
    if (nc[0]) {
        std::vector<int> ids(nc[0]);
        CK(cudaMemcpyAsync(ids.data(), cand, nc[0] * sizeof(int), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        std::sort(ids.begin(), ids.end());
        ids.erase(std::unique(ids.begin(), ids.end()), ids.end());
        const int n = (int)ids.size();
        std::vector<int> firsts;
        for (int b = 0; b < nb; b++) if (vs[b + 1] > vs[b]) firsts.push_back((int)vs[b]);
        std::vector<int> all(ids);
        all.insert(all.end(), firsts.begin(), firsts.end());
        CKS(w.gath.ensure(all.size() * (sizeof(int) + sizeof(vec3d)) + 16));
        vec3d *dpos = w.gath.as<vec3d>();
        int *dids = (int *)(dpos + all.size());
        CK(cudaMemcpyAsync(dids, all.data(), all.size() * sizeof(int), cudaMemcpyHostToDevice, s));
        n2m_launch(k_a_gather, ((int)all.size() + 255) / 256, 256, 0, s, w.pts.as<vec3d>(), dids, (int)all.size(), dpos);
        std::vector<vec3d> pos(all.size());
        CK(cudaMemcpyAsync(pos.data(), dpos, all.size() * sizeof(vec3d), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        int i0 = 0;
        for (int b = 0; b < nb && i0 < n; b++) {
            int i1 = i0;
            while (i1 < n && (unsigned)ids[i1] < vs[b + 1]) i1++;
            if (i1 == i0) continue;
            const int fi = (int)(std::lower_bound(firsts.begin(), firsts.end(), (int)vs[b]) - firsts.begin());
            const vec3d v0 = pos[n + fi];
            const int m = i1 - i0;
            std::vector<float> key(m);
            std::vector<int> srt(m), grp(m, -1);
            for (int k = 0; k < m; k++) { key[k] = (float)d3(v0, pos[i0 + k]); srt[k] = k; }
            std::sort(srt.begin(), srt.end(), [&](int a, int c) {
                return kbits(key[a]) != kbits(key[c]) ? kbits(key[a]) < kbits(key[c]) : ids[i0 + a] < ids[i0 + c];
            });
            int ng = 0;
            for (int k = 0; k < m; k++) {
                const int a = srt[k];
                if (grp[a] >= 0) continue;
                for (int j = k; j < m && (key[srt[j]] - key[a]) < 0.00001f; j++)
                    if (d3(pos[i0 + a], pos[i0 + srt[j]]) < 0.00001f) grp[srt[j]] = ng;
                ng++;
            }
            std::vector<int> gk(ng, INT32_MAX), gl(ng, -1), gs(ng, 0);
            for (int k = 0; k < m; k++) {
                const int g = grp[k];
                gs[g]++;
                gk[g] = std::min(gk[g], ids[i0 + k]);
                if (gl[g] < 0 || ids[i0 + k] > ids[i0 + gl[g]]) gl[g] = k;
            }
            for (int k = 0; k < m; k++) {
                const int g = grp[k];
                if (gs[g] < 2) continue;
                if (ids[i0 + k] != gk[g]) { removed.push_back(ids[i0 + k]); keepv.push_back(gk[g]); }
                else if (gl[g] != k) { ov_id.push_back(ids[i0 + k]); ov_pos.push_back(pos[i0 + gl[g]]); }
            }
            i0 = i1;
        }
    }
    vec3d *pts = w.pts.as<vec3d>();
    WeldMap map;
    unsigned np = nv;
    std::vector<unsigned> vs_new(vs);
    if (!removed.empty()) {
        // ids are grouped by box and ascending within each box, so `removed`
        // is sorted; `ov_id` likewise
        const int nr = (int)removed.size(), no = (int)ov_id.size();
        CKS(w.weld.ensure((size_t)(2 * nr + no + 1) * sizeof(int) + (size_t)(no + 1) * sizeof(vec3d)));
        vec3d *dov = w.weld.as<vec3d>();
        int *drem = (int *)(dov + no + 1), *dkeep = drem + nr, *dovid = dkeep + nr;
        std::vector<int> ri(nr);
        for (int i = 0; i < nr; i++) ri[i] = i;
        std::sort(ri.begin(), ri.end(), [&](int a, int b2) { return removed[a] < removed[b2]; });
        std::vector<int> r2, k2;
        for (int i : ri) { r2.push_back(removed[i]); k2.push_back(keepv[i]); }
        if (no) CK(cudaMemcpyAsync(dov, ov_pos.data(), no * sizeof(vec3d), cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(drem, r2.data(), nr * sizeof(int), cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(dkeep, k2.data(), nr * sizeof(int), cudaMemcpyHostToDevice, s));
        if (no) CK(cudaMemcpyAsync(dovid, ov_id.data(), no * sizeof(int), cudaMemcpyHostToDevice, s));
        np = nv - nr;
        CKS(w.pts2.ensure((size_t)np * sizeof(vec3d)));
        CKS(mesh_apply_weld(pts, (int)nv, drem, nr, dkeep, dovid, dov, no, w.pts2.as<vec3d>(), dw, map, s));
        pts = w.pts2.as<vec3d>();
        for (int b = 0; b <= nb; b++)
            vs_new[b] = vs[b] - (unsigned)(std::lower_bound(r2.begin(), r2.end(), (int)vs[b]) - r2.begin());
        CK(cudaStreamSynchronize(s));
    }
    // ---- degenerate triangles, per-box triangle ranges after compaction
    CKS(w.tris2.ensure((size_t)std::max(nt, 1u) * sizeof(vec3i)));
    CKS(w.ranges.ensure((size_t)(4 * (nb + 1) + 2) * sizeof(unsigned)));
    unsigned *dts = w.ranges.as<unsigned>(), *dkept = dts + (nb + 1), *dvs = dkept + (nb + 1), *dntf = dvs + (nb + 1);
    CK(cudaMemcpyAsync(dts, ts.data(), (nb + 1) * sizeof(unsigned), cudaMemcpyHostToDevice, s));
    CKS(mesh_remove_degenerate(pts, w.tris.as<vec3i>(), (int)nt, map, near, w.tris2.as<vec3i>(), dntf, dw, s));
    if (nt) n2m_launch(k_a_kept, (nb + 128) / 128, 128, 0, s, dts, nb, nt, dw.bits.as<unsigned>(), dw.tiles.as<unsigned>(), dntf,
                       dkept);
    else CK(cudaMemsetAsync(dkept, 0, (nb + 1) * sizeof(unsigned), s));
    std::vector<unsigned> kept(nb + 1);
    CK(cudaMemcpyAsync(kept.data(), dkept, (nb + 1) * sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    const unsigned ntf = kept[nb];
    vec3i *tris = w.tris2.as<vec3i>();
    // ---- HC post-smoothing of all meshes at once (they share no vertex)
    CK(cudaEventRecord(ev[5], s));
    if (o.post_smooth > 0 && np > 0)
        CKS(mesh_smooth_hc(pts, tris, (int)np, (int)ntf, 0.1, 0.5, o.post_smooth, true, hw, sw, s));
    // ---- triangle indices local to their mesh
    CK(cudaMemcpyAsync(dkept, kept.data(), (nb + 1) * sizeof(unsigned), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(dvs, vs_new.data(), (nb + 1) * sizeof(unsigned), cudaMemcpyHostToDevice, s));
    if (ntf) n2m_launch(k_a_localize, pgrid((ntf + 255) / 256, 16), 256, 0, s, tris, ntf, dkept, dvs, nb);
    CKL();
    CK(cudaStreamSynchronize(s));
    out.clear();
    for (int b = 0; b < nb; b++) {
        n2m_atlas_mesh d;
        d.label = boxes[b].label;
        d.status = boxes[b].fail;
        d.nvert = (int)(vs_new[b + 1] - vs_new[b]);
        d.ntri = (int)(kept[b + 1] - kept[b]);
        d.vert_offset = vs_new[b];
        d.tri_offset = kept[b];
        if (!d.status && (d.nvert < 3 || d.ntri < 1)) d.status = N2M_ERR_EMPTY;
        out.push_back(d);
    }
    *d_pts = pts;
    *d_tris = tris;
    *npts = np;
    *ntris = ntf;
    if (ms_stage) {
        for (int i = 0; i < 5; i++) cudaEventElapsedTime(&ms_stage[i], ev[i], ev[i + 1]);
    }
    return N2M_OK;
}
