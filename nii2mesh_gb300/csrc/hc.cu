// hc.cu — laplacian_smoothHC (src/quadric.c:316-394) and its adjoint: neighbour
// gather kernels in FP32 on displacements from the original positions (HC is
// affine-equivariant); border vertices (update_mesh(0), src/quadric.c:184-212)
// keep their input.  The results are compared within a tolerance with the
// reference's FP64 smoothing, so this unit is compiled with FMA contraction
// (the units with bit-exact duties are not).  Also the allocation-free entry
// point n2m_smooth_hc_noalloc.
#include <float.h>

#include <algorithm>

#include "n2m_internal.cuh"

namespace {
inline unsigned gs(size_t n) {
    size_t b = (n + 255) / 256;
    if (b > 152 * 32) b = 152 * 32;
    return b ? (unsigned)b : 1u;
}

// ---- HC smoothing ----------------------------------------------------------------
// A triangle with an index outside [0, np) is skipped here and in k_fill_adj
// (so it never enters the neighbour lists and nothing downstream reads past the
// vertex arrays) and raises *bad; the last sweep then leaves every vertex
// untouched and the entry points report N2M_ERR_BAD_ARGS.
__device__ __forceinline__ bool tri_in_range(const vec3i &T, int np) {
    return (unsigned)T.x < (unsigned)np && (unsigned)T.y < (unsigned)np && (unsigned)T.z < (unsigned)np;
}

__global__ void k_degree(const vec3i *__restrict__ t, int nt, int np, unsigned *deg, unsigned *bad) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
        const vec3i T = t[i];
        if (!tri_in_range(T, np)) {
            *bad = 1u;
            continue;
        }
        atomicAdd(&deg[T.x], 1u);
        atomicAdd(&deg[T.y], 1u);
        atomicAdd(&deg[T.z], 1u);
    }
}

// the two other vertices of every (triangle, slot) reference, in any order within
// the vertex's segment (k_hc_adj sorts it)
__global__ void k_fill_adj(const vec3i *__restrict__ t, int nt, int np, const unsigned *__restrict__ start,
                           unsigned *fill, int2 *adj) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nt; i += gridDim.x * blockDim.x) {
        const vec3i T = t[i];
        if (!tri_in_range(T, np)) continue;
        adj[start[T.x] + atomicAdd(&fill[T.x], 1u)] = make_int2(T.y, T.z);
        adj[start[T.y] + atomicAdd(&fill[T.y], 1u)] = make_int2(T.x, T.z);
        adj[start[T.z] + atomicAdd(&fill[T.z], 1u)] = make_int2(T.x, T.y);
    }
}

// in-place heapsort (neighbour lists that do not fit shared memory: n log n in any order)
__device__ __noinline__ void heapsort_ids(int *a, int n) {
    for (int h = n / 2, e = n; e > 1;) {
        int v;
        if (h > 0) {
            v = a[--h];
        } else {
            v = a[--e];
            a[e] = a[0];
        }
        int r = h;
        for (int c = 2 * r + 1; c < e; c = 2 * r + 1) {
            if (c + 1 < e && a[c + 1] > a[c]) c++;
            if (a[c] <= v) break;
            a[r] = a[c];
            r = c;
        }
        a[r] = v;
    }
}

// One vertex's neighbours.  The smoothing sums the two other vertices of every
// reference, so inside a closed surface each neighbour comes twice: the list
// holds n2 ids that count twice (summed once, doubled), then n1 that count once.
// The first ELL_K of the doubled ids also stand in `ell`, entry k of 32 consecutive
// vertices together, so that a warp reads them in whole lines.
constexpr unsigned ELL_K = 8;
__device__ __forceinline__ size_t ell_at(int i, unsigned k) { return (size_t)(i >> 5) * (32 * ELL_K) + 32 * k + (i & 31); }
struct __align__(16) Meta {
    unsigned at;      // first entry in adj
    unsigned n2, n1;
    float inv;        // 1 / (2 references); 0 when no triangle uses the vertex
};

// Per vertex, once per call: sorts its neighbours (so the sums' order does not
// depend on the atomics that listed them) and pairs them, flags border
// vertices (update_mesh(0), src/quadric.c:184-212: an id seen exactly once
// among a vertex's incident triangles, the vertex's own slots included), and
// computes Lo = L(o) - o in double.  Displacements start at zero, so Lo is
// also the first half of the first iteration: Pn = B = Lo.
// The lists are sorted in shared memory, one column per thread, up to ADJ_S
// entries; longer ones (a fan of more than ADJ_S / 2 triangles) in place, and
// all their entries count once.  Latency-bound (sort, then gathers of the
// neighbours' doubles): 37 us at 250k vertices with cold caches, against 105 us
// for the separate sort, Lo and border kernels that walked triangle references.
constexpr int ADJ_S = 32, ADJ_T = 128;
__global__ void __launch_bounds__(ADJ_T) k_hc_adj(const vec3d *__restrict__ o, const unsigned *__restrict__ start, int np,
                                                  int *adj, int *ell, Meta *meta, unsigned char *border, float4 *Lo,
                                                  float4 *Pn, float4 *B) {
    grid_wait();
    __shared__ int col[ADJ_S][ADJ_T];
    const int tid = threadIdx.x;
    for (int i = blockIdx.x * ADJ_T + tid; i < np; i += gridDim.x * ADJ_T) {
        const unsigned a0 = start[i], d = start[i + 1] - a0, n = 2 * d;
        Meta m = {2 * a0, 0u, 0u, 0.f};
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f);
        if (d) {
            int *g = adj + 2 * (size_t)a0;
            const bool small = n <= (unsigned)ADJ_S;
            if (small) {
                for (unsigned k = 0; k < n; k += 2) {
                    const int2 e = *(const int2 *)(g + k);
                    col[k][tid] = e.x;
                    col[k + 1][tid] = e.y;
                }
                for (unsigned k = 1; k < n; k++) {
                    const int v = col[k][tid];
                    int j = (int)k - 1;
                    for (int w; j >= 0 && (w = col[j][tid]) > v; j--) col[j + 1][tid] = w;
                    col[j + 1][tid] = v;
                }
            } else {
                heapsort_ids(g, (int)n);
            }
            auto id_at = [&](unsigned k) { return small ? col[k][tid] : g[k]; };
            double sx = 0, sy = 0, sz = 0;
            bool self = false;
            for (unsigned k = 0; k < n;) {   // runs of one id
                const int id = id_at(k);
                unsigned e = k + 1;
                while (e < n && id_at(e) == id) e++;
                const vec3d q = o[id];
                const double f = (double)(int)(e - k);
                sx += f * q.x; sy += f * q.y; sz += f * q.z;
                self |= id == i;
                if (e - k == 1 && id != i) border[id] = 1;
                m.n2 += (e - k) >> 1;
                k = e;
            }
            if (d == 1 && !self) border[i] = 1;
            if (small) {
                unsigned w2 = 0, w1 = m.n2;
                for (unsigned k = 0; k < n;) {
                    const int id = col[k][tid];
                    unsigned e = k + 1;
                    while (e < n && col[e][tid] == id) e++;
                    for (unsigned c = (e - k) >> 1; c; c--) {
                        if (w2 < ELL_K) ell[ell_at(i, w2)] = id;
                        g[w2++] = id;
                    }
                    if ((e - k) & 1u) g[w1++] = id;
                    k = e;
                }
                m.n1 = w1 - m.n2;
            } else {
                m.n2 = 0;
                m.n1 = n;
            }
            m.inv = 1.f / (2.f * (float)d);
            const double nn = (double)(int)n;
            lo = make_float4((float)(sx / nn - o[i].x), (float)(sy / nn - o[i].y), (float)(sz / nn - o[i].z), 0.f);
        }
        meta[i] = m;
        Lo[i] = lo;
        Pn[i] = lo;
        B[i] = lo;
    }
}

// Sum of X over the neighbours (W: each scaled by its own .w).  A sweep is bound by the
// latency of its three dependent loads (list, ids, vectors) and by L1: eight ids and
// then their eight 16-byte vectors are in flight at once, one round for the usual valence
// of 6, and the ids come in whole lines from `ell` (per-vertex lists lie 48 bytes apart: a
// warp's load of one id each touched 12 lines).  At 250k vertices with cold caches a
// half-iteration takes 9.4 us; with the ids from the lists it took 10.5, through the
// triangle references (twelve 12-byte vectors behind a fourth dependent load) 14.0.
template <bool W> __device__ __forceinline__ void add_vectors(const float4 *__restrict__ X, const int (&id)[8], float &sx, float &sy, float &sz) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = id[u] >= 0 ? __ldg(X + id[u]) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; u++) {
        if (W) {
            sx += v[u].x * v[u].w; sy += v[u].y * v[u].w; sz += v[u].z * v[u].w;
        } else {
            sx += v[u].x; sy += v[u].y; sz += v[u].z;
        }
    }
}
template <bool W>
__device__ __forceinline__ void add_ids(const float4 *__restrict__ X, const int *__restrict__ p, unsigned n, float &sx,
                                        float &sy, float &sz) {
    for (unsigned k = 0; k < n; k += 8) {
        int id[8];
#pragma unroll
        for (int u = 0; u < 8; u++) id[u] = k + u < n ? __ldg(p + k + u) : -1;
        add_vectors<W>(X, id, sx, sy, sz);
    }
}
struct Lists {
    const int *adj, *ell;
};
template <bool W>
__device__ __forceinline__ float3 sum_neighbours(const float4 *__restrict__ X, const Lists &l, int i, const Meta &m) {
    float ax = 0.f, ay = 0.f, az = 0.f;
    const int *__restrict__ e = l.ell + ell_at(i, 0);
    int id[8];
    static_assert(ELL_K == 8, "one round");
#pragma unroll
    for (int u = 0; u < 8; u++) id[u] = (unsigned)u < m.n2 ? __ldg(e + 32 * u) : -1;
    add_vectors<W>(X, id, ax, ay, az);
    if (m.n2 > ELL_K) add_ids<W>(X, l.adj + m.at + ELL_K, m.n2 - ELL_K, ax, ay, az);
    ax += ax; ay += ay; az += az;
    if (m.n1) add_ids<W>(X, l.adj + m.at + m.n2, m.n1, ax, ay, az);
    return make_float3(ax, ay, az);
}
__device__ __forceinline__ Meta load_meta(const Meta *__restrict__ meta, int i) {
    const uint4 u = __ldg((const uint4 *)meta + i);
    return Meta{u.x, u.y, u.z, __uint_as_float(u.w)};
}

// first half of an HC iteration: Pn = L(p) - o, B = Pn - (1-alpha) Q
__global__ void __launch_bounds__(128) k_hc_a(const float4 *__restrict__ P, const float4 *__restrict__ Lo,
                                              const Meta *__restrict__ meta, Lists lists, int np,
                                              float alpha1, float4 *Pn, float4 *B) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const Meta m = load_meta(meta, i);
        const float4 q = P[i], lo = Lo[i];
        float4 pn = q;
        if (m.inv != 0.f) {
            const float3 l = sum_neighbours<false>(P, lists, i, m);
            pn = make_float4(lo.x + l.x * m.inv, lo.y + l.y * m.inv, lo.z + l.z * m.inv, 0.f);
        }
        Pn[i] = pn;
        B[i] = make_float4(pn.x - alpha1 * q.x, pn.y - alpha1 * q.y, pn.z - alpha1 * q.z, 0.f);
    }
}

// second half: P = Pn - (beta B + (1-beta) L(B)); the last one (o set) moves the
// vertices instead: o += P, except border vertices when locked, and none at all
// when a triangle index was out of range
__global__ void __launch_bounds__(128) k_hc_b(const float4 *__restrict__ Pn, const float4 *__restrict__ B,
                                              const Meta *__restrict__ meta, Lists lists, int np,
                                              float beta, float beta1, float4 *P, vec3d *o,
                                              const unsigned char *__restrict__ border, bool lock,
                                              const unsigned *__restrict__ bad) {
    grid_wait();
    if (o && *bad) return;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const Meta m = load_meta(meta, i);
        const float4 b = B[i], pn = Pn[i];
        float3 lb = make_float3(b.x, b.y, b.z);
        if (m.inv != 0.f) {
            lb = sum_neighbours<false>(B, lists, i, m);
            lb = make_float3(lb.x * m.inv, lb.y * m.inv, lb.z * m.inv);
        }
        const float3 d = make_float3(pn.x - (beta * b.x + beta1 * lb.x), pn.y - (beta * b.y + beta1 * lb.y),
                                     pn.z - (beta * b.z + beta1 * lb.z));
        if (!o) {
            P[i] = make_float4(d.x, d.y, d.z, 0.f);
        } else if (!(lock && border[i])) {
            o[i].x += (double)d.x; o[i].y += (double)d.y; o[i].z += (double)d.z;
        }
    }
}

// ---- HC adjoint ------------------------------------------------------------------------
// One iteration is p' = A p + B o with L the (row-normalised) neighbour mean:
//   A = beta(1-alpha) I + (1-beta)(2-alpha) L - (1-beta) L^2,  B = alpha beta I + alpha(1-beta) L.
// Backward: lambda = dL/dp_K; per iteration g_o += B^T lambda, lambda = A^T lambda; finally
// g_o += lambda (p_0 = o).  L^T y at j sums y_i / num_i over the same (triangle, slot)
// references (the neighbour relation is symmetric); isolated vertices are identity rows.
// The vectors carry 1 / num_i in .w, so a gather brings both.
__global__ void k_hcT_init(const float3 *__restrict__ g, const unsigned char *__restrict__ border,
                           const Meta *__restrict__ meta, int np, bool lock, float4 *lam, float3 *go) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const bool b = lock && border[i];
        const float3 v = g[i];
        const float inv = meta[i].inv;
        lam[i] = b ? make_float4(0.f, 0.f, 0.f, inv) : make_float4(v.x, v.y, v.z, inv);
        go[i] = b ? v : make_float3(0.f, 0.f, 0.f);
    }
}

// t1 = L^T lam
__global__ void __launch_bounds__(128) k_hcT_a(const float4 *__restrict__ lam, const Meta *__restrict__ meta,
                                               Lists lists, int np, float4 *t1) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const Meta m = load_meta(meta, i);
        float4 r = lam[i];
        if (m.inv != 0.f) {
            const float3 s = sum_neighbours<true>(lam, lists, i, m);
            r = make_float4(s.x, s.y, s.z, m.inv);
        }
        t1[i] = r;
    }
}

// t2 = L^T t1; go += ab*lam + a1b*t1; lam = c0*lam + c1*t1 - c2*t2 (added to go by the last iteration)
__global__ void __launch_bounds__(128) k_hcT_b(float4 *lam, const float4 *__restrict__ t1, const Meta *__restrict__ meta,
                                               Lists lists, float3 *go, int np, float ab, float a1b,
                                               float c0, float c1, float c2, bool last) {
    grid_wait();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const Meta m = load_meta(meta, i);
        const float4 l = lam[i], u = t1[i];
        float3 v = make_float3(u.x, u.y, u.z);
        if (m.inv != 0.f) v = sum_neighbours<true>(t1, lists, i, m);
        float3 g = go[i];
        g.x += ab * l.x + a1b * u.x; g.y += ab * l.y + a1b * u.y; g.z += ab * l.z + a1b * u.z;
        const float4 n = make_float4(c0 * l.x + c1 * u.x - c2 * v.x, c0 * l.y + c1 * u.y - c2 * v.y,
                                     c0 * l.z + c1 * u.z - c2 * v.z, l.w);
        if (last) {
            g.x += n.x; g.y += n.y; g.z += n.z;
        } else {
            lam[i] = n;
        }
        go[i] = g;
    }
}

// the buffers of one smoothing: `zero` (start, fill, bad, border) is cleared first
struct HcBufs {
    unsigned *start, *fill, *bad;
    unsigned char *border;
    size_t zero_bytes;
    int *adj, *ell;
    Meta *meta;
    float4 *P, *Q, *B, *Lo;
};
size_t hc_zero_layout(int np, void *base, HcBufs &h) {
    h.start = (unsigned *)base;              // np + 1 counts, scanned to offsets
    h.fill = h.start + np + 1;
    h.bad = h.fill + np;
    h.border = (unsigned char *)(h.bad + 1);
    return h.zero_bytes = (size_t)(2 * (size_t)np + 2) * sizeof(unsigned) + (size_t)np;
}
inline unsigned sweep_grid(int np) { return (unsigned)std::max(1, std::min((np + 127) / 128, 152 * 64)); }

n2m_status hc_count(const vec3i *d_tris, int np, int nt, const HcBufs &h, cudaStream_t s) {
    CK(cudaMemsetAsync(h.start, 0, h.zero_bytes, s));
    n2m_launch(k_degree, gs(nt), 256, 0, s, d_tris, nt, np, h.start, h.bad);
    CKL();
    return N2M_OK;
}
// everything after the scan of the degrees; iter >= 1
n2m_status hc_run(vec3d *d_pts, const vec3i *d_tris, int np, int nt, double alpha, double beta, int iter, bool lock_edges,
                  const HcBufs &h, cudaStream_t s) {
    n2m_launch(k_fill_adj, gs(nt), 256, 0, s, d_tris, nt, np, h.start, h.fill, (int2 *)h.adj);
    const unsigned g = sweep_grid(np);
    n2m_launch(k_hc_adj, g, ADJ_T, 0, s, d_pts, h.start, np, h.adj, h.ell, h.meta, h.border, h.Lo, h.Q, h.B);
    const float a1 = (float)(1.0 - alpha), b = (float)beta, b1 = (float)(1.0 - beta);
    for (int it = 0; it < iter; it++) {
        if (it) n2m_launch(k_hc_a, g, 128, 0, s, h.P, h.Lo, h.meta, Lists{h.adj, h.ell}, np, a1, h.Q, h.B);
        n2m_launch(k_hc_b, g, 128, 0, s, h.Q, h.B, h.meta, Lists{h.adj, h.ell}, np, b, b1, h.P, it + 1 == iter ? d_pts : nullptr, h.border,
                   lock_edges, h.bad);
    }
    CKL();
    return N2M_OK;
}
HcBufs hc_bufs(const HcWork &w, int np) {
    HcBufs h;
    hc_zero_layout(np, w.zero.p, h);
    h.adj = w.adj.as<int>();
    h.ell = w.ell.as<int>();
    h.meta = w.meta.as<Meta>();
    h.P = w.P.as<float4>();
    h.Q = w.Q.as<float4>();
    h.B = w.B.as<float4>();
    h.Lo = w.Lo.as<float4>();
    return h;
}
}  // namespace

n2m_status mesh_smooth_hc(vec3d *d_pts, const vec3i *d_tris, int np, int nt, double alpha, double beta, int iter,
                          bool lock_edges, HcWork &w, ScanWork &sw, cudaStream_t s) {
    if (np <= 0 || iter <= 0) return N2M_OK;
    HcBufs h;
    CKS(w.zero.ensure(hc_zero_layout(np, nullptr, h)));
    CKS(w.adj.ensure((size_t)6 * (nt > 0 ? nt : 1) * sizeof(int)));
    CKS(w.ell.ensure(((size_t)np + 31) / 32 * 32 * ELL_K * sizeof(int)));
    CKS(w.meta.ensure((size_t)np * sizeof(Meta)));
    CKS(w.P.ensure((size_t)np * sizeof(float4)));
    CKS(w.Q.ensure((size_t)np * sizeof(float4)));
    CKS(w.B.ensure((size_t)np * sizeof(float4)));
    CKS(w.Lo.ensure((size_t)np * sizeof(float4)));
    h = hc_bufs(w, np);
    CKS(hc_count(d_tris, np, nt, h, s));
    CKS(scan_u32(h.start, (size_t)np + 1, h.start + np, sw, s));   // start[np] receives the total as well
    return hc_run(d_pts, d_tris, np, nt, alpha, beta, iter, lock_edges, h, s);
}

n2m_status mesh_smooth_hc_check(HcWork &w, int np, int iter, cudaStream_t s) {
    if (np <= 0 || iter <= 0) return N2M_OK;
    unsigned bad = 0;
    CK(cudaMemcpyAsync(&bad, hc_bufs(w, np).bad, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (bad) {
        n2m_set_error("HC smoothing: a triangle index is outside [0, nvert); the vertices were left unchanged");
        return N2M_ERR_BAD_ARGS;
    }
    return N2M_OK;
}

n2m_status mesh_smooth_hc_backward(int np, double alpha, double beta, int iter, bool lock_edges, HcWork &w,
                                   const float3 *d_g, float3 *d_go, cudaStream_t s) {
    // adjacency and border flags are the forward's; its vectors serve as scratch (P lambda, Q t1)
    const HcBufs h = hc_bufs(w, np);
    const unsigned g = sweep_grid(np);
    n2m_launch(k_hcT_init, gs(np), 256, 0, s, d_g, h.border, h.meta, np, lock_edges, h.P, d_go);
    const float al = (float)alpha, be = (float)beta;
    const float ab = al * be, a1b = al * (1.f - be);
    const float c0 = be * (1.f - al), c1 = (1.f - be) * (2.f - al), c2 = 1.f - be;
    for (int it = 0; it < iter; it++) {
        n2m_launch(k_hcT_a, g, 128, 0, s, h.P, h.meta, Lists{h.adj, h.ell}, np, h.Q);
        n2m_launch(k_hcT_b, g, 128, 0, s, h.P, h.Q, h.meta, Lists{h.adj, h.ell}, d_go, np, ab, a1b, c0, c1, c2, it + 1 == iter);
    }
    CKL();
    return N2M_OK;
}

// ---- allocation-free HC smoothing ---------------------------------------------------
// For callers that cannot call cudaMalloc: code running inside another
// framework's captured or allocation-controlled region, or a host program that
// owns all device memory through its own pool.  The scratch of the HC
// smoothing (neighbour lists, displacement buffers, flags) lives in one
// file-scope device array of fixed size, so the entry point allocates nothing.
// Limits: N2M_NOALLOC_MAX_VERTS vertices and N2M_NOALLOC_MAX_TRIS triangles
// (about 22 MB, held by every GPU that loads the library until exit).
namespace {
constexpr size_t NA_V = N2M_NOALLOC_MAX_VERTS, NA_T = N2M_NOALLOC_MAX_TRIS;
constexpr size_t na_align(size_t b) { return (b + 255) & ~(size_t)255; }
constexpr size_t NA_ADJ = na_align((2 * NA_V + 2) * 4 + NA_V);   // after the counts, cursors and flags
constexpr size_t NA_META = NA_ADJ + na_align(NA_T * 6 * 4);
constexpr size_t NA_P = NA_META + na_align(NA_V * 16);
constexpr size_t NA_Q = NA_P + na_align(NA_V * 16);
constexpr size_t NA_B = NA_Q + na_align(NA_V * 16);
constexpr size_t NA_LO = NA_B + na_align(NA_V * 16);
constexpr size_t NA_ELL = NA_LO + na_align(NA_V * 16);
constexpr size_t NA_TOTAL = NA_ELL + na_align((NA_V + 31) / 32 * 32 * ELL_K * 4);

static __device__ __align__(256) unsigned char g_noalloc_scratch[NA_TOTAL];

// exclusive scan of n <= NA_V + 1 counts in one CTA (n is small by construction)
__global__ void __launch_bounds__(1024) k_scan_small(unsigned *d, int n) {
    grid_wait();
    __shared__ unsigned part[1024];
    __shared__ unsigned carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const unsigned v = i < n ? d[i] : 0u;
        part[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < 1024; o <<= 1) {
            const unsigned t = threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
            __syncthreads();
            part[threadIdx.x] += t;
            __syncthreads();
        }
        if (i < n) d[i] = carry + part[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry += part[1023];
        __syncthreads();
    }
}
}  // namespace

// Every call looks up the device address of the scratch array on the current
// device (cudaGetSymbolAddress allocates nothing), so the address is never
// stale, e.g. after the caller reset the device.  The first call on a device
// may load the library's device code; make it before any stream capture.
extern "C" n2m_status n2m_smooth_hc_noalloc(vec3d *d_verts, const vec3i *d_tris, int nvert, int ntri, double alpha,
                                            double beta, int iter, bool lock_edges, void *stream) {
    if (nvert < 0 || ntri < 0 || (nvert > 0 && !d_verts) || (ntri > 0 && !d_tris)) {
        n2m_set_error("n2m_smooth_hc_noalloc: bad arguments");
        return N2M_ERR_BAD_ARGS;
    }
    if ((size_t)nvert > NA_V || (size_t)ntri > NA_T) {
        n2m_set_error("n2m_smooth_hc_noalloc: mesh of %d vertices / %d triangles exceeds the fixed scratch "
                      "(max %d vertices, %d triangles)", nvert, ntri, N2M_NOALLOC_MAX_VERTS, N2M_NOALLOC_MAX_TRIS);
        return N2M_ERR_TOO_LARGE;
    }
    if (nvert == 0 || iter <= 0) return N2M_OK;
    unsigned char *base = nullptr;
    CK(cudaGetSymbolAddress((void **)&base, g_noalloc_scratch));
    cudaStream_t s = (cudaStream_t)stream;
    // the array keeps the previous call's contents; hc_count clears what must start at zero
    HcBufs h;
    hc_zero_layout(nvert, base, h);
    h.adj = (int *)(base + NA_ADJ);
    h.meta = (Meta *)(base + NA_META);
    h.P = (float4 *)(base + NA_P);
    h.Q = (float4 *)(base + NA_Q);
    h.B = (float4 *)(base + NA_B);
    h.Lo = (float4 *)(base + NA_LO);
    h.ell = (int *)(base + NA_ELL);
    CKS(hc_count(d_tris, nvert, ntri, h, s));
    n2m_launch(k_scan_small, 1, 1024, 0, s, h.start, nvert + 1);
    CKS(hc_run(d_verts, d_tris, nvert, ntri, alpha, beta, iter, lock_edges, h, s));
    // the validity flag comes back through pageable host memory: a plain copy, no allocation
    unsigned h_bad = 0;
    CK(cudaMemcpyAsync(&h_bad, h.bad, sizeof(unsigned), cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
    if (h_bad) {
        n2m_set_error("n2m_smooth_hc_noalloc: a triangle index is outside [0, nvert); the vertices were left unchanged");
        return N2M_ERR_BAD_ARGS;
    }
    return N2M_OK;
}
