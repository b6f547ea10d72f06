// n2m_internal.cuh — shared declarations of the CUDA implementation.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>
#include <string>
#include <vector>

#include "../../include/n2m_gpu.h"

#define N2M_FLT_EPS 1.19209290e-07f

// Grids are bounded by multiples of 152, the SMs of a GB300 (and LZ_SLOTS in deflate.cu is what one
// of them holds): on another number of SMs the kernels are correct, their grids no longer fit it.

// ---- error plumbing ---------------------------------------------------------
void n2m_set_error(const char *fmt, ...);
#define CK(call)                                                                          \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            n2m_set_error("%s:%d %s: %s", __FILE__, __LINE__, #call, cudaGetErrorString(e_)); \
            (void)cudaGetLastError();   /* not left for the next call */                  \
            return e_ == cudaErrorMemoryAllocation ? N2M_ERR_OOM : N2M_ERR_CUDA;          \
        }                                                                                 \
    } while (0)
#define CKS(st)                                   \
    do {                                          \
        n2m_status s_ = (st);                     \
        if (s_ != N2M_OK) return s_;              \
    } while (0)
#define CKL()  CK(cudaGetLastError())

// process-wide count of kernel launches (reported by n2m_kernel_launches)
extern std::atomic<long long> g_n2m_launches;

// Every kernel is launched with n2m_launch and begins with grid_wait().  The launch lets
// the next kernel of the stream be set up while this one's last blocks leave (no kernel
// releases its successor earlier, so two kernels' blocks never run side by side), and
// grid_wait() returns once everything before it in the stream is complete and visible.
// A call is a chain of 30 to 45 kernels of a few microseconds, and the gap between two of
// them counts: 64^3 spheres 423 -> 382 us, brain with Otsu level 808 -> 755, 128^3 fit
// 1328 -> 1198, HC drop-in 933 -> 842.  Letting successors start as soon as all blocks of
// a kernel run was slower (brain 776, HC 1000 us: waiting blocks take slots).
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline void n2m_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t shared, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = shared;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    (void)cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);   // an error is found by CKL()
    g_n2m_launches.fetch_add(1, std::memory_order_relaxed);
}

// bytes of a context's pinned buffer for small readbacks
constexpr size_t N2M_READBACK = 16384;

// ---- grow-only device buffers -----------------------------------------------
struct DevBuf {
    void *p = nullptr;
    size_t cap = 0;
    n2m_status ensure(size_t bytes);
    void release();
    template <class T> T *as() const { return reinterpret_cast<T *>(p); }
};

// ---- ordered-int encoding of floats for atomicMin/atomicMax ------------------
__device__ __forceinline__ int f2ord(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
inline int f2ord_host(float f) {
    int i;
    memcpy(&i, &f, 4);
    return i >= 0 ? i : i ^ 0x7fffffff;
}
__host__ __device__ __forceinline__ float ord2f(int i) {
    int j = i >= 0 ? i : i ^ 0x7fffffff;
#ifdef __CUDA_ARCH__
    return __int_as_float(j);
#else
    float f;
    memcpy(&f, &j, 4);
    return f;
#endif
}

// Reductions produced by the volume passes (device-resident, read back once).
struct VolStats {
    int vmin, vmax;          // ordered-int min/max of the volume
    int lo[3], hi[3];        // bbox of voxels >= iso (unpadded, inclusive)
    unsigned nonfinite;      // NaN/Inf voxels
    unsigned masked;         // voxels the labelling set to the minimum (run_labelling)
};

// ---- kernels' host launchers (stream-ordered, no syncs) ----------------------
// smooth.cu
// A host volume copied to `in` slab by slab on the `copy` stream while the
// x pass of the slabs already copied runs (the three-pass path only).
constexpr int N2M_STAGE_SLABS = 16;
struct StagedInput {
    const float *host = nullptr;
    cudaStream_t copy = nullptr;
    cudaEvent_t ev[N2M_STAGE_SLABS + 1] = {};
};
// tmp: one volume of scratch; stage: see StagedInput (may be null)
n2m_status launch_smooth(const float *in, float *out, float *tmp, int nx, int ny, int nz, float iso, VolStats *st,
                         cudaStream_t s, const StagedInput *stage = nullptr);
// whether launch_smooth can take a StagedInput for this volume
bool smooth_can_stage(int nx, int ny, int nz);

// Pre-smooth with exact rounding on demand (smooth.cu): od_approx smooths the
// whole volume approximately (one fused FP32 pass, rigorous error bound), lists
// the voxels whose sign against iso it cannot decide and leaves the range of each
// task; od_resolve gives those voxels, and every voxel that can be the volume's
// minimum or maximum (or of a plateau of those, some), their exact values, which
// completes w.st (exact range and bbox in its vs).  Once the host has read w.st, od_check
// says whether the caller has to run launch_smooth instead (a non-finite or huge input, more
// undecided voxels than the list holds, a plateau whose value does not follow from the raw volume).
// Marching cubes marks the voxels whose values it reads in `need` (mcwords.cuh:
// k_words, with an OdRepair): the ends of the edges the surface crosses and the
// corners of ambiguous cubes; od_repair writes the reference's exact value at every
// marked voxel of `out`.
enum : unsigned { OD_FALLBACK = 1u, OD_TIMEOUT = 2u };
struct OdStats {
    VolStats vs;             // bbox of decided voxels >= iso; exact range after od_resolve
    unsigned flags;          // final after od_resolve
    unsigned cnt[3];         // undecided, min candidates, max candidates
    int umin, lmax;          // ordered: smallest task min + B, largest task max - B
    unsigned done;           // blocks of od_resolve that are through, when a list of candidates is too short
    int rlo[4], rhi[4];      // then, ordered: raw range of the voxels in the face layers of at least 0 .. 3 axes
};
struct OdLists {
    unsigned *unc, *cmin, *cmax;   // voxels
    unsigned *cnt;
    unsigned cap;
    unsigned *vsign;         // sign bitmap of the smoothed volume (see OdWork)
    float4 *range;           // per task of pass A {min, max, B, -}
    unsigned wv, nys;        // the bitmap's words per row, groups of 8 rows per slice
};
struct OdWork {
    DevBuf st, need, list, lcnt;   // st: OdStats, the lists of undecided voxels and range candidates, the tasks' ranges
    // bit x & 31 of word od_vsign_word(x, y, z): the smoothed value of voxel (x, y, z)
    // minus iso is above -FLT_EPSILON (Lewiner's sign before edge darkening), or with
    // od_resolve's at_or_above, the value is >= iso (the complement of oldcubes'
    // sign); exact for every voxel once od_resolve has run
    DevBuf vsign;
    unsigned cap = 0;
};
// What meshify's labelling does to each voxel (src/meshify.c:330-342), for the values
// marching cubes reads: voxels of K (bit x & 31 of word (z*ny + y)*W + x/32) are raised
// to iso when fill; voxels outside KD (K and its dilation) are the minimum mn.  S: the
// sign bitmap of the result.  KD and S are null when the volume itself was labelled.
struct LabelPost {
    const unsigned *K, *KD, *S;
    unsigned W;
    float mn, iso;
    bool fill, largest;
};
struct OdRepair {
    const float *in;         // the raw volume
    float *tmp1, *tmp2;      // exact x and y pass values (written at marked voxels only)
    float *out;              // the approximately smoothed volume, exact where marked
    int dim[3];
    OdWork *w;
    const LabelPost *post = nullptr;   // the volume was labelled: the repaired values get the same treatment
};
// the sign bitmap's word of voxel (x, y, z): the 8 row words of one 32 x 8 tile of a
// slice are adjacent (one 32-byte sector, written at once by pass A)
__host__ __device__ __forceinline__ size_t od_vsign_word(unsigned x, unsigned y, unsigned z, unsigned wv, unsigned nys) {
    return (((size_t)z * nys + (y >> 3)) * wv + (x >> 5)) * 8u + (y & 7u);
}
// whether the on-demand path applies: at least 5 voxels along each axis, fewer than 2^32
bool od_eligible(int nx, int ny, int nz);
// bytes of od_approx's scratch (the input with rows of a multiple of 16 bytes, if its own are not); at least the volume's
size_t od_scratch(const float *in, int nx, int ny, int nz);
n2m_status od_approx(const float *in, float *out, int nx, int ny, int nz, float iso, float *scratch, OdWork &w, cudaStream_t s);
n2m_status od_resolve(const float *in, float *out, int nx, int ny, int nz, float iso, OdWork &w, cudaStream_t s,
                      bool at_or_above = false);
n2m_status od_check(const OdStats &h, bool *fallback);
// the cleared mark bitmap: bit x & 31 of word (z*ny + y)*ceil(nx/32) + x/32
n2m_status od_marks(OdWork &w, const int dim[3], unsigned **need, cudaStream_t s);
n2m_status od_repair(const OdRepair &r, cudaStream_t s);
// transposed pre-smooth: g_img = Sx^T Sy^T Sz^T g (tmp: one volume of scratch)
n2m_status launch_smooth_adjoint(const float *g, float *tmp, float *out, int nx, int ny, int nz, cudaStream_t s);
// (z0: slice of vol in the whole volume)
n2m_status launch_stats(const float *vol, int nx, int ny, int nz, float iso, bool minmax, VolStats *st,
                        cudaStream_t s, int z0 = 0);
void stats_init_host(VolStats *h);

// scan.cu: exclusive scan in place; total -> *d_total
struct ScanWork {
    DevBuf part;
};
n2m_status scan_u32(unsigned *d, size_t n, unsigned *d_total, ScanWork &w, cudaStream_t s);

// label.cu
struct LabelWork {
    DevBuf lab, mask, keep, cnt, edge, rc, misc, list, wlist, cs, filled, shell;
};
// meshify's labelling of vol: the kept set in *post, and with only_largest (and mn
// clearly below iso) also what follows from it without writing the volume: signs, bbox
// and count of masked voxels (st).  Otherwise (post->S null), and when st says that no
// voxel was masked, lab_write labels the volume in place and gives its range and bbox.
// vsign (may be null): a sign bitmap (OdWork::vsign with od_resolve's at_or_above) to
// take the mask from; at_or_above: which sign S holds (value >= iso, for oldcubes);
// skip (may be null): a device word that, if not zero, leaves the labelling undone (it was
// queued before the smoothing was known to hold; its results are not read then)
// (the minimum, post->mn, is the caller's to fill in)
n2m_status run_labelling(const float *vol, int nx, int ny, int nz, float iso, bool only_largest, bool fill_bubbles,
                         bool at_or_above, LabelWork &w, VolStats *st, cudaStream_t s, const unsigned *vsign, const unsigned *skip,
                         LabelPost *post);
n2m_status lab_write(float *vol, int nx, int ny, int nz, const LabelPost &P, VolStats *st, cudaStream_t s);
// the labelling's effect on the marked voxels of vol (marks as od_marks lays them out)
n2m_status lab_apply(float *vol, int nx, int ny, int nz, const unsigned *need, const LabelPost &P, cudaStream_t s);
// bwlabel() semantics on a float volume (nonzero = foreground); *d_nl gets the label count
n2m_status run_bwlabel(float *vol, int nx, int ny, int nz, int conn, bool only_largest, bool fill_bubbles,
                       LabelWork &w, ScanWork &sw, int *d_nl, cudaStream_t s);

// decode.cu: NIfTI voxel cast (bytes per voxel 0 = unsupported datatype)
int nifti_bytes_per_voxel(int datatype);
n2m_status launch_cast(const void *d_raw, int datatype, float slope, float inter, long long n, float *d_out,
                       cudaStream_t s);

// deflate.cu: gzip / zlib / raw deflate of n bytes at d_src (4-byte aligned, n + 8
// readable bytes); the stream goes to w.out, its length to *out_len (synchronizes
// once to size the output).  deflate_check reads back the emitter's self-check.
struct DeflateWork {
    DevBuf tok, info, hist, codes, hdr, sizes, misc, out;
    int lz_slots = 0;                                       // chunks the match finder keeps in flight
    int huff_slots = 0;                                     // warps the code builder keeps in flight
    void *side = nullptr, *ev_in = nullptr, *ev_ck = nullptr;   // checksum stream and its events
};
size_t deflate_bound(size_t n);
void deflate_release(DeflateWork &w);
n2m_status deflate_device(const void *d_src, size_t n, int container, DeflateWork &w, ScanWork &sw, cudaStream_t s,
                          size_t *out_len);
n2m_status deflate_check(DeflateWork &w, cudaStream_t s);

// writers.cu: the bytes save_mesh() writes, assembled in device memory
struct WriterWork {
    DevBuf mt, mp, pack, pack2, lens, flag, out;
    DeflateWork df;
    void *host = nullptr;   // pinned staging for file writes
    size_t host_cap = 0;
};
int mesh_format_of(const char *fnm);   // N2M_FMT_*, or -1 (save_mesh appends ".mz3")
const char *file_ext(const char *fnm);  // where strip_ext cuts the name
n2m_status encode_mesh_device(int format, const vec3i *d_t, const vec3d *d_p, int nt, int np, bool gz, WriterWork &w,
                              ScanWork &sw, cudaStream_t s, const unsigned char **d_out, size_t *len);

// isolevel.cu: setThreshold (Otsu on the robust range) of a device volume
struct ThresholdWork {
    DevBuf buf, table;
    std::vector<double> P;
};
n2m_status isolevel_otsu(const float *d_img, long long nvox, int mode123, ThresholdWork &w, cudaStream_t s,
                         float *result, void *pinned);

// mc.cu
struct McGrid {
    const float *vol;        // processed volume (before edge darkening)
    int dim[3];              // volume dims
    int lo[3];               // grid origin in the volume
    int n[3];                // grid size (NX, NY, NZ)
    float iso, edge_max, pad_val;   // pad_val = float(min' - iso)
};
struct McWork {
    DevBuf signs;            // sign words of the grid
    DevBuf words;            // per active word {x, y, z crossing masks, vertex offset}
    DevBuf act;              // active words in order {word, triangle offset, c-vertex offset, -}
    DevBuf cnt, sub;         // counting scratch (mcwords.cuh: Out)
};
struct McCounts {
    unsigned nv_edge, nt, nc, nactive;
};
// What marching cubes and the stages after it leave for the host, read back at once.
// The kernels from the emit on take the counts from here, so that they can be queued
// before the host knows them; each does nothing if the mesh does not fit its buffers.
constexpr int MARCH_CAND = 256;
struct MarchOut {
    uint4 tot;                  // edge vertices, triangles, c-vertices, active words
    unsigned ncand, nccand;     // weld candidates: edge vertices, c-vertices
    unsigned kept;              // triangles left by the degenerate filter, if it ran
    unsigned pad;
    vec3d first;                // with candidates: the first vertex, and the first MARCH_CAND
    vec3d cand_pos[MARCH_CAND]; // candidates
    int cand_id[MARCH_CAND];
};
struct MeshRoom {
    unsigned nv, nt;            // vertices and triangles the buffers hold
    __host__ __device__ bool fits(uint4 t) const {
        return (unsigned long long)t.x + t.z <= nv && t.y <= nt;
    }
};
// post: what a labelling did to the volume (its signs are post->S), repair: the volume
// was smoothed approximately (without post its signs are repair->w->vsign); with
// either, the voxels whose values are needed are marked after the sign pass and put
// right before any value is read.  od: the marks' and the repair's buffers.
n2m_status mc_count(const McGrid &g, int variant, McWork &w, uint4 *d_total, cudaStream_t s, OdWork &od,
                    const OdRepair *repair = nullptr, const LabelPost *post = nullptr);
n2m_status mc_emit(const McGrid &g, int variant, McWork &w, MarchOut *d_out, const MeshRoom &room, vec3d *d_pts, vec3i *d_tris,
                   int *d_cand, int cand_cap, unsigned *d_near, cudaStream_t s);
n2m_status mc_backward(const McGrid &g, int variant, McWork &w, const McCounts &c, const float3 *d_gv, float *d_gs,
                       cudaStream_t s);
n2m_status mc_ccand_scan(const vec3d *d_pts, int np, const int *d_ccand, int nccand, int *d_cand,
                         unsigned *d_ncand, int cand_cap, cudaStream_t s);

// oldcubes.cu
// as mc_count (the sign bitmaps must then hold value >= iso)
n2m_status oc_count(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso, float edge_max,
                    McWork &w, uint4 *d_total, cudaStream_t s, OdWork &od, const OdRepair *repair = nullptr,
                    const LabelPost *post = nullptr);
n2m_status oc_emit(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso, float edge_max,
                    McWork &w, MarchOut *d_out, const MeshRoom &room, vec3d *d_pts, vec3i *d_tris, int *d_cand,
                    int cand_cap, unsigned *d_near, cudaStream_t s);
// the copies of the ncand weld candidates in the reference's triangle soup: every
// corner 3*t + c naming one, into d_out (at most cap; *d_count = how many there
// are); d_bits: nv bits of scratch
n2m_status oc_copies(const vec3i *d_tris, int nt, int nv, const int *d_cand, int ncand, unsigned *d_bits,
                     unsigned *d_out, unsigned *d_count, unsigned cap, cudaStream_t s);
// the vertex id each listed corner names and the position the cube that emitted
// its triangle interpolates for it (needs oc_count's words of the same grid)
n2m_status oc_copy_positions(const float *vol, const int dim[3], const int lo[3], const int hi[3], float iso,
                             float edge_max, const McWork &w, unsigned nactive, const vec3i *d_tris, const unsigned *d_q,
                             int n, int *d_vid, vec3d *d_pos, cudaStream_t s);

// mesh.cu
constexpr int DEG_TILE = 1024;   // triangles of a tile of the degenerate filter
struct DegWork {
    DevBuf bits;    // a bit per triangle: kept
    DevBuf tiles;   // kept triangles before each tile of DEG_TILE; counts per tile and group
    DevBuf rank;    // of the weld
    DevBuf near;    // a bit per vertex: close to a grid point
};
// what the weld does to vertex ids: per 32 vertices {removed ones, removed before them}
// (null: no weld); the k-th removed one merges into keep[k]
struct WeldMap {
    const uint2 *rank = nullptr;
    const int *keep = nullptr;
};
n2m_status mesh_apply_weld(const vec3d *d_pts, int np, const int *d_removed, int nrem, const int *d_keep,
                           const int *d_ov_id, const vec3d *d_ov_pos, int nov, vec3d *d_out, DegWork &w, WeldMap &map,
                           cudaStream_t s);
// Vertices of marching cubes closer than this to a grid point are marked for the
// degenerate filter (mesh.cu: k_deg_count).  Lewiner's distance is that of the stored
// coordinate, already rounded (at 2^15 a float is a 256th of a voxel): an unmarked vertex is
// where it is stored, at least this far from the ends of its edge, and so the bound on the area
// holds for the stored triangle.  (Oldcubes takes the fraction along the edge: its positions are
// doubles.)  Coordinates below 2^22: mc33::frac_dist rounds to integers there.
constexpr float NEAR_CORNER = 1.f / 512;
__device__ __forceinline__ void mark_near(unsigned *near, int id) {
    if (near) atomicOr(near + (id >> 5), 1u << (id & 31));
}
// d_tris_in is renumbered in place if the weld removed vertices; d_near: the marks by raw id, or null
n2m_status mesh_remove_degenerate(const vec3d *d_pts, vec3i *d_tris_in, int nt, const WeldMap &weld, const unsigned *d_near,
                                  vec3i *d_tris_out, unsigned *d_nt_out, DegWork &w, cudaStream_t s);
// the same, queued before the host knows the counts: if the mesh fits `room` and nothing can be welded, the filter runs
// (out->kept), else the weld candidates are left in *out
n2m_status mesh_after_emit(const vec3d *d_pts, vec3i *d_tris_in, const MeshRoom &room, const int *d_cand, int cand_cap,
                           const unsigned *d_near, vec3i *d_tris_out, MarchOut *d_out, DegWork &w, cudaStream_t s);
// only the candidates
n2m_status mesh_weld_candidates(const vec3d *d_pts, const MeshRoom &room, const int *d_cand, int cand_cap, MarchOut *d_out,
                                cudaStream_t s);
struct HcWork {
    DevBuf zero;              // degrees / offsets, cursors, the bad-index flag, border flags
    DevBuf adj, ell, meta;    // neighbour lists, their first entries by 32 vertices, per-vertex heads
    DevBuf P, Q, B, Lo;       // displacements
};
// Triangles with an index outside [0, np) are skipped and flagged; the flag
// makes the last kernel leave d_pts unchanged.  mesh_smooth_hc_check waits for
// the stream and returns N2M_ERR_BAD_ARGS when the flag was raised (entry
// points that take the caller's triangles call it; meshify's own meshes are
// valid by construction).
n2m_status mesh_smooth_hc(vec3d *d_pts, const vec3i *d_tris, int np, int nt, double alpha, double beta, int iter,
                          bool lock_edges, HcWork &w, ScanWork &sw, cudaStream_t s);
n2m_status mesh_smooth_hc_check(HcWork &w, int np, int iter, cudaStream_t s);
// adjoint of mesh_smooth_hc (uses the neighbour lists and border flags the forward left in w)
n2m_status mesh_smooth_hc_backward(int np, double alpha, double beta, int iter, bool lock_edges, HcWork &w,
                                   const float3 *d_g, float3 *d_go, cudaStream_t s);
// grad of raw (pre-weld) vertices from grad of welded vertices
n2m_status mesh_weld_backward(const float3 *d_go, int nv_raw, const int *d_removed, int nrem,
                              const int *d_ov_id, const int *d_ov_src, int nov, float3 *d_graw, cudaStream_t s);
n2m_status mesh_apply_sform(vec3d *d_pts, vec3i *d_tris, int np, int nt, const float sx[4], const float sy[4],
                            const float sz[4], cudaStream_t s);

// atlas.cu
#include <vector>
struct AtlasWork {
    McWork mc;
    DevBuf cnt, bb, boxes, arena, mask, keep, fill, shell, wbox, list, wlist, lab, edge, ucnt, subbox, tot, pts, pts2, tris, tris2,
        cand, gath, weld, ranges;
};
n2m_status atlas_hist(const short *d_lab, const int dim[3], AtlasWork &w, cudaStream_t s, int *maxlab,
                      std::vector<unsigned> &cnt, std::vector<int> &bb);
n2m_status atlas_binarize(const short *d_lab, long long n, int label, float *out, cudaStream_t s);
n2m_status atlas_offset_tris(vec3i *t, int n, int off, cudaStream_t s);
n2m_status atlas_batched(const short *d_lab, const int dim[3], const n2m_options &o, AtlasWork &w, ScanWork &sw,
                         DegWork &dw, HcWork &hw, cudaStream_t s, std::vector<n2m_atlas_mesh> &out, vec3d **d_pts,
                         vec3i **d_tris, int64_t *npts, int64_t *ntris, float *ms_stage);
