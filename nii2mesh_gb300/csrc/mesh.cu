// mesh.cu — per-mesh stages after marching cubes:
//   * weld fix-up (src/meshify.c:45-106): applies the merges the host decided
//     for the few near-grid-point candidates (vertex compaction; the triangles
//     are renumbered by the degenerate filter);
//   * remove_degenerate_triangles (src/meshify.c:113-168): FP32 area filter
//     with a rigorous error margin, the reference's FP64 predicate for the
//     rest, stable compaction;
//   * the weld's adjoint (a welded vertex's gradient back to its raw vertex);
//   * apply_sform (src/meshify.c:1021-1045).
// laplacian_smoothHC is in hc.cu.
#include <float.h>

#include "n2m_internal.cuh"

namespace {
// ---- weld -------------------------------------------------------------------
__device__ __forceinline__ int lower_bound(const int *a, int n, int v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int m = (lo + hi) >> 1;
        if (a[m] < v) lo = m + 1;
        else hi = m;
    }
    return lo;
}

// removed[k] (sorted) merges into keep[k]; override ids (sorted) take pos.  rank, per 32
// vertices: which of them are removed, and how many before them.
__global__ void __launch_bounds__(256) k_weld_verts(const vec3d *__restrict__ in, int np, const int *__restrict__ removed,
                                                    int nrem, const int *__restrict__ ov_id,
                                                    const vec3d *__restrict__ ov_pos, int nov, vec3d *__restrict__ out,
                                                    uint2 *rank) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (((unsigned)np + 31u) & ~31u); i += gridDim.x * blockDim.x) {
        const int r = lower_bound(removed, nrem, (int)i);
        const bool gone = r < nrem && removed[r] == (int)i;
        const unsigned b = __ballot_sync(0xffffffffu, gone);
        if ((i & 31u) == 0) rank[i / 32] = make_uint2(b, (unsigned)r);
        if (gone || i >= (unsigned)np) continue;
        const int o = lower_bound(ov_id, nov, (int)i);
        out[i - r] = (o < nov && ov_id[o] == (int)i) ? ov_pos[o] : in[i];
    }
}

// vertex v after the weld; the ranks of consecutive vertices share cache lines (a search
// in the removed ids per corner is a chain of ten loads)
__device__ __forceinline__ int welded(int v, uint2 k, const WeldMap &m) {
    int r = (int)k.y + __popc(k.x & ((1u << (v & 31)) - 1u));
    if (k.x >> (v & 31) & 1u) {
        v = m.keep[r];
        k = __ldg(m.rank + v / 32);
        r = (int)k.y + __popc(k.x & ((1u << (v & 31)) - 1u));
    }
    return v - r;
}

// ---- degenerate triangles --------------------------------------------------------
__device__ __forceinline__ double dist_d(vec3d a, vec3d b) {
    const double dx = __dsub_rn(a.x, b.x), dy = __dsub_rn(a.y, b.y), dz = __dsub_rn(a.z, b.z);
    return __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
}

// the reference predicate, operation for operation (src/meshify.c:119-144)
__device__ bool degenerate_ref(vec3d A, vec3d B, vec3d C) {
    const double l = dist_d(A, B), m = dist_d(A, C), n = dist_d(B, C);
    const double c = fmin(fmin(l, m), n), a = fmax(fmax(l, m), n);
    const double b = __dsub_rn(__dsub_rn(__dadd_rn(__dadd_rn(l, m), n), a), c);
    const double cab = __dsub_rn(c, __dsub_rn(a, b));
    if (cab <= 0.0) return true;
    const double q = __dmul_rn(__dmul_rn(__dmul_rn(__dadd_rn(a, __dadd_rn(b, c)), cab), __dadd_rn(c, __dsub_rn(a, b))),
                               __dadd_rn(a, __dsub_rn(b, c)));
    return __dmul_rn(0.25, __dsqrt_rn(q)) < (double)FLT_EPSILON;
}

// Fast path: the area from an FP32 cross product of (double) edge vectors, minus a
// bound on its rounding error, exceeding 4e-7 (> 3x FLT_EPSILON) proves the
// triangle is kept under the reference predicate.
// float value of d if d is exactly a float (zero or normal), by bit assembly:
// the F2F conversion issues on the FP64 pipe, a small fraction of the integer
// rate on this part
__device__ __forceinline__ bool d2f_exact(double d, float &f) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(d);
    const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
    const unsigned long long m = b & 0xfffffffffffffull;
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    if (e == 0 && m == 0) { f = __uint_as_float(sign); return true; }
    if ((m & 0x1fffffffull) || e < 897u || e > 1150u) return false;   // low bits set or outside the normal float range
    f = __uint_as_float(sign | ((e - 896u) << 23) | (unsigned)(m >> 29));
    return true;
}

__device__ __forceinline__ bool surely_kept(vec3d A, vec3d B, vec3d C) {
    float ax, ay, az, bx, by, bz, qx, qy, qz;
    float ux, uy, uz, vx, vy, vz;
    if (d2f_exact(A.x, ax) & d2f_exact(A.y, ay) & d2f_exact(A.z, az) & d2f_exact(B.x, bx) & d2f_exact(B.y, by) &
        d2f_exact(B.z, bz) & d2f_exact(C.x, qx) & d2f_exact(C.y, qy) & d2f_exact(C.z, qz)) {
        // float coordinates: the FP32 difference is the double difference rounded to float
        ux = bx - ax; uy = by - ay; uz = bz - az;
        vx = qx - ax; vy = qy - ay; vz = qz - az;
    } else {
        ux = (float)(B.x - A.x); uy = (float)(B.y - A.y); uz = (float)(B.z - A.z);
        vx = (float)(C.x - A.x); vy = (float)(C.y - A.y); vz = (float)(C.z - A.z);
    }
    const float cx = uy * vz - uz * vy, cy = uz * vx - ux * vz, cz = ux * vy - uy * vx;
    const float cr = sqrtf(cx * cx + cy * cy + cz * cz);
    const float nu = sqrtf(ux * ux + uy * uy + uz * uz), nv = sqrtf(vx * vx + vy * vy + vz * vz);
    return 0.5f * (cr - 1e-6f * nu * nv) > 4e-7f && isfinite(cr);
}

constexpr int CB = 256;          // threads of a CTA
constexpr int DT = DEG_TILE;     // triangles of a CTA
constexpr int DG = 64;           // tiles of a group
static_assert(DT == 4 * CB && DT == 32 * 32, "four triangles per thread, a warp of words");

// Kept triangles as bits, and their number per tile and group of tiles; the weld's
// renumbering, if there was one, on the way.  Gathering three 24-byte vertices per
// triangle bounded this (L1 wavefronts), and nearly every triangle is far from
// degenerate.  NEAR: marching cubes marked the vertices closer than NEAR_CORNER to
// a grid point (and all cell-centre vertices).  A triangle whose corners are on three edges
// of a cube, none of them marked, has an area above 3e-6, far above FLT_EPSILON, so only
// triangles with a marked corner (1 %) are looked at; they are listed, so that they share
// warps.  The bits of neighbouring vertices share sectors.  Without marks (vertices from
// elsewhere) every triangle is, four consecutive ones per lane, which share most
// vertices.  512^3 CT (7.6 M triangles): flags of 4 bytes, a triangle per lane and a pass of
// its own for the renumbering took 93 + 61 us, the general path here 126 (the whole filter
// with the copy 164), with the marks the filter takes 111; oldcubes (4.1 M) 132 -> 61.
template <bool NEAR>
__device__ __forceinline__ void deg_count_tile(unsigned tile, const vec3d *__restrict__ p, vec3i *t, int nt, const WeldMap &m,
                                               const unsigned *__restrict__ near, unsigned *bits, unsigned *tile_cnt,
                                               unsigned *group_cnt) {
    __shared__ unsigned kept[DT / 32], nslow;
    __shared__ unsigned short slow[DT];
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned i0 = tile * DT + 4u * tid;
    const int n = i0 < (unsigned)nt ? (int)min(4u, (unsigned)nt - i0) : 0;
    if (tid == 0) nslow = 0;
    __syncthreads();
    int v[12];
    if (n == 4) {
        const int4 *q = (const int4 *)(t + i0);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const int4 x = q[k];
            v[4 * k] = x.x; v[4 * k + 1] = x.y; v[4 * k + 2] = x.z; v[4 * k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 12; k++) v[k] = k < 3 * n ? ((const int *)(t + i0))[k] : 0;
    }
    unsigned look = 0;   // corners of triangles to look at
    if (NEAR && n) {
#pragma unroll
        for (int k = 0; k < 12; k++) look |= (__ldg(near + v[k] / 32) >> (v[k] & 31) & 1u) << k;
    }
    if (m.rank && n) {
        uint2 q[12];
#pragma unroll
        for (int k = 0; k < 12; k++) q[k] = __ldg(m.rank + v[k] / 32);
#pragma unroll
        for (int k = 0; k < 12; k++) v[k] = k < 3 * n ? welded(v[k], q[k], m) : 0;
        if (n == 4) {
            int4 *q4 = (int4 *)(t + i0);
#pragma unroll
            for (int k = 0; k < 3; k++) q4[k] = make_int4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        } else {
#pragma unroll
            for (int k = 0; k < 12; k++)
                if (k < 3 * n) ((int *)(t + i0))[k] = v[k];
        }
    }
    unsigned keep = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (k < n) {
            if (NEAR ? !(look >> (3 * k) & 7u) : surely_kept(p[v[3 * k]], p[v[3 * k + 1]], p[v[3 * k + 2]])) keep |= 1u << k;
            else slow[atomicAdd(&nslow, 1u)] = (unsigned short)(4 * tid + k);
        }
    unsigned w = keep << (4 * (lane & 7));   // eight lanes make a word
    for (int o = 1; o < 8; o <<= 1) w |= __shfl_xor_sync(0xffffffffu, w, o);
    if ((lane & 7) == 0) kept[tid / 8] = w;
    __syncthreads();
    for (unsigned k = tid; k < nslow; k += CB) {
        const int i = slow[k];
        const vec3i T = t[tile * DT + i];
        if ((NEAR && surely_kept(p[T.x], p[T.y], p[T.z])) || !degenerate_ref(p[T.x], p[T.y], p[T.z])) atomicOr(&kept[i / 32], 1u << (i & 31));
    }
    __syncthreads();
    if (tid < 32) {
        w = kept[tid];
        bits[tile * (DT / 32) + tid] = w;
        const unsigned sum = __reduce_add_sync(0xffffffffu, __popc(w));
        if (tid == 0) {
            tile_cnt[tile] = sum;
            atomicAdd(&group_cnt[tile / DG], sum);
        }
    }
}

// the weld's candidates for the host
__device__ __forceinline__ void give_candidates(const vec3d *__restrict__ p, const int *__restrict__ cand, MarchOut *mo) {
    const unsigned n = mo->ncand;
    for (unsigned k = threadIdx.x; k < min(n, (unsigned)MARCH_CAND); k += blockDim.x) {
        mo->cand_id[k] = cand[k];
        mo->cand_pos[k] = p[cand[k]];
    }
    if (threadIdx.x == 0) mo->first = p[0];
}

__global__ void __launch_bounds__(CB) k_weld_candidates(const vec3d *__restrict__ p, MeshRoom room, const int *__restrict__ cand,
                                                        int cap, MarchOut *mo) {
    grid_wait();
    if (mo->ncand && mo->ncand <= (unsigned)cap && room.fits(mo->tot)) give_candidates(p, cand, mo);
}

// with mo the number of triangles is its count; nothing is done if the mesh did not fit or has to be welded first
template <bool NEAR>
__global__ void __launch_bounds__(CB, 4) k_deg_count(const vec3d *__restrict__ p, vec3i *t, int nt, WeldMap m,
                                                     const unsigned *__restrict__ near, unsigned *bits, unsigned *tile_cnt,
                                                     unsigned *group_cnt, MarchOut *mo, MeshRoom room, const int *__restrict__ cand,
                                                     int cap) {
    grid_wait();
    if (mo) {
        if (!room.fits(mo->tot)) return;
        if (mo->ncand | mo->nccand) {
            if (blockIdx.x == 0 && mo->ncand && mo->ncand <= (unsigned)cap) give_candidates(p, cand, mo);
            return;
        }
        nt = (int)mo->tot.y;
    }
    const unsigned tiles = ((unsigned)nt + DT - 1) / DT;
    for (unsigned tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        deg_count_tile<NEAR>(tile, p, t, nt, m, near, bits, tile_cnt, group_cnt);
        __syncthreads();   // the lists are reused by the next tile
    }
}

// The kept triangles in order.  A tile adds up the groups and tiles before it by itself
// (a scan in between was three launches); a tile without a degenerate triangle,
// nearly every one, is a plain copy.  tile_off: kept triangles before each tile.
// 512^3 CT: 48 us with a lane per 12-byte record.
__device__ __forceinline__ void deg_compact_tile(int tile, int tiles, const vec3i *__restrict__ t, int nt,
                                                 const unsigned *__restrict__ bits, const unsigned *__restrict__ tile_cnt,
                                                 const unsigned *__restrict__ group_cnt, unsigned *tile_off, vec3i *out,
                                                 unsigned *nt_out) {
    __shared__ unsigned wsum[CB / 32], pre[DT / 32];
    __shared__ int stage[3 * DT];
    const int g = tile / DG, tid = threadIdx.x;
    unsigned s = 0;
    for (int k = tid; k < g; k += CB) s += group_cnt[k];
    if (tid < tile - g * DG) s += tile_cnt[g * DG + tid];
    s = __reduce_add_sync(0xffffffffu, s);
    if ((tid & 31) == 0) wsum[tid >> 5] = s;
    __syncthreads();
    unsigned off = 0;
    for (int k = 0; k < CB / 32; k++) off += wsum[k];
    const int have = min(DT, nt - tile * DT);
    const unsigned cnt = tile_cnt[tile];
    if (tid == 0) {
        tile_off[tile] = off;
        if (tile == tiles - 1) *nt_out = off + cnt;
    }
    const int *src = (const int *)(t + (size_t)tile * DT);
    int *dst = (int *)(out + off);
    if (cnt == (unsigned)have) {
#pragma unroll 4
        for (int k = tid; k < 3 * have; k += CB) dst[k] = src[k];
        return;
    }
    if (tid < 32) {
        const unsigned c = __popc(bits[tile * (DT / 32) + tid]);
        unsigned incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned x = __shfl_up_sync(0xffffffffu, incl, o);
            if (tid >= o) incl += x;
        }
        pre[tid] = incl - c;
    }
    __syncthreads();
    for (int i = tid; i < have; i += CB) {
        const unsigned w = bits[tile * (DT / 32) + i / 32];
        if (!(w >> (i & 31) & 1u)) continue;
        const unsigned at = pre[i / 32] + __popc(w & ((1u << (i & 31)) - 1u));
        for (int c = 0; c < 3; c++) stage[3 * at + c] = src[3 * i + c];
    }
    __syncthreads();
    for (int k = tid; k < 3 * (int)cnt; k += CB) dst[k] = stage[k];
}

__global__ void __launch_bounds__(CB) k_deg_compact(const vec3i *__restrict__ t, int nt, const unsigned *__restrict__ bits,
                                                    const unsigned *__restrict__ tile_cnt, const unsigned *__restrict__ group_cnt,
                                                    unsigned *tile_off, vec3i *out, unsigned *nt_out, const MarchOut *mo,
                                                    MeshRoom room) {
    grid_wait();
    if (mo) {
        if (!room.fits(mo->tot) || (mo->ncand | mo->nccand)) return;
        nt = (int)mo->tot.y;
    }
    const int tiles = (int)(((unsigned)nt + DT - 1) / DT);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        deg_compact_tile(tile, tiles, t, nt, bits, tile_cnt, group_cnt, tile_off, out, nt_out);
        __syncthreads();   // the stage is reused by the next tile
    }
}

// raw vertex gradient: every kept raw vertex receives its welded vertex's
// gradient, except that a merged group's gradient goes to the member whose
// position it kept
__global__ void k_weld_back(const float3 *__restrict__ go, int nv_raw, const int *__restrict__ removed, int nrem,
                            const int *__restrict__ ov_id, const int *__restrict__ ov_src, int nov, float3 *graw) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nv_raw; i += gridDim.x * blockDim.x) {
        const int r = lower_bound(removed, nrem, i);
        if (r < nrem && removed[r] == i) continue;
        const int o = lower_bound(ov_id, nov, i);
        const int src = (o < nov && ov_id[o] == i) ? ov_src[o] : i;
        const float3 g = go[i - r];
        atomicAdd(&graw[src].x, g.x);
        atomicAdd(&graw[src].y, g.y);
        atomicAdd(&graw[src].z, g.z);
    }
}

__global__ void k_sform(vec3d *p, int np, double a0, double a1, double a2, double a3, double b0, double b1, double b2,
                        double b3, double c0, double c1, double c2, double c3) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const vec3d v = p[i];
        p[i].x = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(v.x, a0), __dmul_rn(v.y, a1)), __dmul_rn(v.z, a2)), a3);
        p[i].y = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(v.x, b0), __dmul_rn(v.y, b1)), __dmul_rn(v.z, b2)), b3);
        p[i].z = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(v.x, c0), __dmul_rn(v.y, c1)), __dmul_rn(v.z, c2)), c3);
    }
}

__global__ void k_flip(vec3i *t, int nt) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
        const int x = t[i].x;
        t[i].x = t[i].y;
        t[i].y = x;
    }
}

inline unsigned gs(size_t n) {
    size_t b = (n + 255) / 256;
    if (b > 152 * 32) b = 152 * 32;
    return b ? (unsigned)b : 1u;
}
}  // namespace

n2m_status mesh_apply_weld(const vec3d *d_pts, int np, const int *d_removed, int nrem, const int *d_keep,
                           const int *d_ov_id, const vec3d *d_ov_pos, int nov, vec3d *d_out, DegWork &w, WeldMap &map,
                           cudaStream_t s) {
    CKS(w.rank.ensure(((size_t)np + 31) / 32 * sizeof(uint2)));
    map.rank = w.rank.as<uint2>();
    map.keep = d_keep;
    n2m_launch(k_weld_verts, gs(np), 256, 0, s, d_pts, np, d_removed, nrem, d_ov_id, d_ov_pos, nov, d_out, w.rank.as<uint2>());
    CKL();
    return N2M_OK;
}

namespace {
struct DegBufs {
    unsigned *bits, *off, *cnt, *grp;
};
// buffers of the filter for nt triangles; the groups' counters are cleared
n2m_status deg_buffers(long long nt, DegWork &w, cudaStream_t s, DegBufs &b) {
    const long long tiles = std::max(1ll, (nt + DT - 1) / DT), groups = (tiles + DG - 1) / DG;
    CKS(w.bits.ensure((size_t)tiles * (DT / 32) * sizeof(unsigned)));
    CKS(w.tiles.ensure(((size_t)2 * tiles + groups) * sizeof(unsigned)));
    b.bits = w.bits.as<unsigned>();
    b.off = w.tiles.as<unsigned>();
    b.cnt = b.off + tiles;
    b.grp = b.cnt + tiles;
    CK(cudaMemsetAsync(b.grp, 0, (size_t)groups * sizeof(unsigned), s));
    return N2M_OK;
}
}  // namespace

n2m_status mesh_remove_degenerate(const vec3d *d_pts, vec3i *d_tris_in, int nt, const WeldMap &weld, const unsigned *d_near,
                                  vec3i *d_tris_out, unsigned *d_nt_out, DegWork &w, cudaStream_t s) {
    if (nt == 0) {
        CK(cudaMemsetAsync(d_nt_out, 0, sizeof(unsigned), s));
        return N2M_OK;
    }
    const int tiles = (int)(((long long)nt + DT - 1) / DT);
    DegBufs b;
    CKS(deg_buffers(nt, w, s, b));
    const MeshRoom all{0u, 0u};
    if (d_near) n2m_launch(k_deg_count<true>, tiles, CB, 0, s, d_pts, d_tris_in, nt, weld, d_near, b.bits, b.cnt, b.grp, nullptr,
                           all, nullptr, 0);
    else n2m_launch(k_deg_count<false>, tiles, CB, 0, s, d_pts, d_tris_in, nt, weld, nullptr, b.bits, b.cnt, b.grp, nullptr, all,
                    nullptr, 0);
    n2m_launch(k_deg_compact, tiles, CB, 0, s, d_tris_in, nt, b.bits, b.cnt, b.grp, b.off, d_tris_out, d_nt_out, nullptr, all);
    CKL();
    return N2M_OK;
}

n2m_status mesh_after_emit(const vec3d *d_pts, vec3i *d_tris_in, const MeshRoom &room, const int *d_cand, int cand_cap,
                           const unsigned *d_near, vec3i *d_tris_out, MarchOut *d_out, DegWork &w, cudaStream_t s) {
    DegBufs b;
    CKS(deg_buffers(room.nt, w, s, b));
    // the buffers may be much larger than this mesh: no more blocks than stay resident
    const unsigned g = std::max(1u, std::min((room.nt + DT - 1) / DT, 152u * 6u));
    const WeldMap none;
    if (d_near) n2m_launch(k_deg_count<true>, g, CB, 0, s, d_pts, d_tris_in, 0, none, d_near, b.bits, b.cnt, b.grp, d_out, room,
                           d_cand, cand_cap);
    else n2m_launch(k_deg_count<false>, g, CB, 0, s, d_pts, d_tris_in, 0, none, nullptr, b.bits, b.cnt, b.grp, d_out, room, d_cand,
                    cand_cap);
    n2m_launch(k_deg_compact, g, CB, 0, s, d_tris_in, 0, b.bits, b.cnt, b.grp, b.off, d_tris_out, &d_out->kept, d_out, room);
    CKL();
    return N2M_OK;
}

n2m_status mesh_weld_candidates(const vec3d *d_pts, const MeshRoom &room, const int *d_cand, int cand_cap, MarchOut *d_out,
                                cudaStream_t s) {
    n2m_launch(k_weld_candidates, 1, CB, 0, s, d_pts, room, d_cand, cand_cap, d_out);
    CKL();
    return N2M_OK;
}

n2m_status mesh_weld_backward(const float3 *d_go, int nv_raw, const int *d_removed, int nrem,
                              const int *d_ov_id, const int *d_ov_src, int nov, float3 *d_graw, cudaStream_t s) {
    CK(cudaMemsetAsync(d_graw, 0, (size_t)nv_raw * sizeof(float3), s));
    n2m_launch(k_weld_back, gs(nv_raw), 256, 0, s, d_go, nv_raw, d_removed, nrem, d_ov_id, d_ov_src, nov, d_graw);
    CKL();
    return N2M_OK;
}

n2m_status mesh_apply_sform(vec3d *d_pts, vec3i *d_tris, int np, int nt, const float sx[4], const float sy[4],
                            const float sz[4], cudaStream_t s) {
    n2m_launch(k_sform, gs(np), 256, 0, s, d_pts, np, sx[0], sx[1], sx[2], sx[3], sy[0], sy[1], sy[2], sy[3], sz[0], sz[1],
               sz[2], sz[3]);
    const double px = (double)(sx[0] + sx[1] + sx[2]), py = (double)(sy[0] + sy[1] + sy[2]),
                 pz = (double)(sz[0] + sz[1] + sz[2]);
    const float det = (float)(px * py * pz);
    if (det < 0.0) n2m_launch(k_flip, gs(nt), 256, 0, s, d_tris, nt);
    CKL();
    return N2M_OK;
}

