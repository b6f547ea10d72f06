// label.cu — connected-component labelling for meshify's largest-cluster and
// bubble-fill options (src/bwlabel.c:429-543, src/meshify.c:323-342) and the
// drop-in bwlabel().
//
// Runs, not voxels.  The class masks are bit words (bit x & 31 of word
// row*W + x/32, W = ceil(nx/32) words per row), and union-find links exist
// only at the first voxel of every run along x: a run is one set of voxels
// for any connectivity, so a component is a set of runs.  Two runs in
// neighbouring rows are united once per overlap (the contact whose left
// neighbours do not also touch), hooking the larger root under the smaller,
// so the root of a component is its first voxel in raster order: that is how
// the reference numbers labels (first appearance) and breaks size ties (lowest
// label wins).  Flattening, face contacts, bubble filling, component sizes and
// the kept component all work per run, and the labelled volume itself is never
// written: what marching cubes needs of it follows from the kept set (k_lab_shell).
//
// A word's thread finds the start of the run of any of its bits by itself: the
// last start within the word, or, for a run that began in an earlier word, the
// entry k_run_starts left for the word (one max-scan per row and class; walking or
// scanning the rows again in every kernel made them bound by instructions).
//
// All of it waits on scattered loads of links (L2 latency) and on unions, not on
// bandwidth: the first contact of a run is its parent without a union, pointers are
// jumped to roots before the other contacts are looked at, and the kernels run over
// lists of runs or words, so that no lane idles.  512^3 CT volume (18-connected
// foreground, 6-connected background): contacts 775 -> 252 us, of it 145 us for the
// foreground; the sizes 91 -> 48 us where noise makes a million runs (int16 scan);
// the whole call 2184 -> 1538 us with the volume left unwritten.
#include <algorithm>

#include "n2m_internal.cuh"
#include "runs.cuh"
#include "smooth_core.cuh"
#include "uf.cuh"

namespace {
using namespace uf;
using namespace runs;

struct LD {
    int nx, ny, nz;
    long long nxy, n;
    unsigned W;       // words per row
    unsigned nrows;   // ny * nz
    unsigned nwords;  // W * nrows
    int seg;          // lanes per row in the row kernels
};

__device__ __forceinline__ unsigned valid_bits(const LD &d, unsigned w) {
    const int x0 = (int)w * 32;
    return x0 + 32 <= d.nx ? FULL : (1u << (d.nx - x0)) - 1u;
}

// foreground bits (want 1) or background bits (want 0) of word w of row r
__device__ __forceinline__ unsigned class_word(const unsigned *B, const LD &d, unsigned r, unsigned w, unsigned want) {
    const unsigned b = B[(size_t)r * d.W + w];
    return want ? b : ~b & valid_bits(d, w);
}

// Class bits of the volume: value >= iso (meshify's mask), or value != 0
// (bwlabel's).  A warp takes whole rows, 16 words at a time in flight.
__global__ void __launch_bounds__(256) k_lab_bits(const float *__restrict__ vol, LD d, float iso, bool nonzero,
                                                  unsigned *B) {
    grid_wait();
    constexpr int K = 16;
    const int lane = threadIdx.x & 31;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < d.nrows; r += (gridDim.x * blockDim.x) >> 5) {
        const float *rp = vol + (long long)r * d.nx;
        unsigned *out = B + (size_t)r * d.W;
        for (unsigned w0 = 0; w0 < d.W; w0 += K) {
            float v[K];
#pragma unroll
            for (int k = 0; k < K; k++) {
                const int x = (int)(w0 + k) * 32 + lane;
                v[k] = w0 + k < d.W && x < d.nx ? __ldg(rp + x) : 0.f;
            }
            unsigned mine = 0;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const int x = (int)(w0 + k) * 32 + lane;
                const unsigned m = __ballot_sync(FULL, x < d.nx && (nonzero ? v[k] != 0.0f : v[k] >= iso));
                if (lane == k) mine = m;
            }
            if (lane < K && w0 + lane < d.W) out[w0 + lane] = mine;
        }
    }
}

// Class bits from a sign bitmap (bit = value >= iso; OdWork::vsign layout:
// wv = W words per row, the 8 row words of a 32 x 8 tile of a slice adjacent)
__global__ void k_lab_bits_vsign(const unsigned *__restrict__ vsign, LD d, unsigned nys, unsigned *B) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < d.nwords; i += gridDim.x * blockDim.x) {
        const unsigned r = i / d.W, w = i - r * d.W, z = r / (unsigned)d.ny, y = r - z * (unsigned)d.ny;
        B[i] = __ldg(vsign + od_vsign_word(w * 32u, y, z, d.W, nys)) & valid_bits(d, w);
    }
}

// Contact directions of a run with the rows before it: row k (0: its own, 1: (y-1, z), 2: (y, z-1), 3: (y-1, z-1),
// 4: (y+1, z-1)) at x offset dx; 6-connectivity takes the first two, 18- the first eight, 26- all
__host__ __device__ constexpr int dir_k(int i) { return (int)(0x443343221121ull >> (4 * i) & 15ull); }
__host__ __device__ constexpr int dir_x(int i) { return (int)(0x202011202011ull >> (4 * i) & 15ull) - 1; }
__host__ __device__ constexpr int ndirs(int nnb) { return nnb == 3 ? 2 : (nnb == 9 ? 8 : 12); }
static_assert(dir_k(0) == 1 && dir_k(1) == 2 && dir_k(2) == 1 && dir_k(3) == 1 && dir_k(4) == 2 && dir_k(5) == 2 && dir_k(6) == 3 &&
                  dir_k(7) == 4 && dir_k(8) == 3 && dir_k(9) == 3 && dir_k(10) == 4 && dir_k(11) == 4, "contact rows");
static_assert(dir_x(0) == 0 && dir_x(1) == 0 && dir_x(2) == -1 && dir_x(3) == 1 && dir_x(4) == -1 && dir_x(5) == 1 && dir_x(6) == 0 &&
                  dir_x(7) == 0 && dir_x(8) == -1 && dir_x(9) == 1 && dir_x(10) == -1 && dir_x(11) == 1, "contact offsets");

// cs[i]: where (x) the run that reaches into word i from the word before it starts (-1: no run start before the word).
// `seg` lanes (a power of two, one word per lane) per row, rows of more than 32 words in chunks of 32.
__global__ void __launch_bounds__(256) k_run_starts(const unsigned *__restrict__ B, LD d, unsigned want, int *cs) {
    grid_wait();
    const int lane = threadIdx.x & 31, seg = d.seg, li = lane & (seg - 1);
    const unsigned rpw = 32u / (unsigned)seg, rsub = (unsigned)lane / (unsigned)seg;
    const unsigned nw = (gridDim.x * blockDim.x) >> 5;
    for (unsigned rb = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * rpw; rb < d.nrows; rb += nw * rpw) {
        const unsigned r = rb + rsub;
        int cst = -1;
        unsigned cwd = 0;
        for (unsigned c0 = 0; c0 < d.W; c0 += (unsigned)seg) {
            const unsigned w = c0 + (unsigned)li;
            const bool ok = r < d.nrows && w < d.W;
            const int start = run_before(ok ? class_word(B, d, r, w, want) : 0u, (int)w * 32, li, seg, cst, cwd);
            if (ok) cs[(size_t)r * d.W + w] = start;
        }
    }
}

// a word of a row with the words around it
struct Word {
    unsigned c, pc, nc;   // this word, the one before, the one after (0 outside the row)
    unsigned r, w;
    __device__ __forceinline__ unsigned starts() const { return c & ~((c << 1) | (pc >> 31)); }
    // bits x whose voxel x + dx is in the class
    __device__ __forceinline__ unsigned shifted(int dx) const {
        return dx == 0 ? c : dx == 1 ? (c >> 1) | (nc << 31) : dx == -1 ? (c << 1) | (pc >> 31) : (c << 2) | (pc >> 30);
    }
    // voxel index of the start of the run that voxel b (-1 .. 32 of this word) belongs to
    __device__ __forceinline__ int run(const LD &d, const int *__restrict__ cs, int b) const {
        const int x0 = (int)w * 32;
        int x;
        if (b > 31 && !(c >> 31)) x = x0 + 32;
        else {
            x = b < 0 ? -1 : last_start(starts(), x0, min(b, 31));
            if (x < 0) x = __ldg(cs + (size_t)r * d.W + w);
        }
        return (int)((long long)r * d.nx + x);
    }
};
__device__ __forceinline__ Word load_word(const unsigned *__restrict__ B, const LD &d, unsigned r, unsigned w, unsigned want) {
    return Word{class_word(B, d, r, w, want), w ? class_word(B, d, r, w - 1, want) : 0u,
                w + 1 < d.W ? class_word(B, d, r, w + 1, want) : 0u, r, w};
}
// word w of row r and of the NR - 1 rows before it that touch it
template <int NNB>
struct Around {
    static constexpr int NR = NNB == 3 ? 3 : 5;
    Word q[NR];
    __device__ __forceinline__ void load(const unsigned *__restrict__ B, const LD &d, unsigned want, const Word &own) {
        constexpr int RY[5] = {0, -1, 0, -1, 1}, RZ[5] = {0, 0, -1, -1, -1};
        const int z = (int)(own.r / (unsigned)d.ny), y = (int)(own.r - (unsigned)z * (unsigned)d.ny);
        q[0] = own;
#pragma unroll
        for (int k = 1; k < NR; k++) {
            const int yy = y + RY[k], zz = z + RZ[k];
            const bool ok = yy >= 0 && zz >= 0 && yy < d.ny && zz < d.nz;
            q[k] = ok ? load_word(B, d, (unsigned)zz * (unsigned)d.ny + (unsigned)yy, own.w, want) : Word{0u, 0u, 0u, 0u, own.w};
        }
    }
};

// The run starts of the class, and the words that hold any of it, as lists (their order
// is free): the kernels that follow wait on memory most of the time, and by rows of
// words only a few lanes of a warp had a run (512^3: 0.8 M background runs in 4.2 M
// words, a foreground in a tenth of them).
constexpr int LIST_K = 2;   // words per thread (8: a block for 2048 words left most SMs of a small volume idle)
static_assert(256 * LIST_K * 16 < 65536, "a block's run starts and words share one 32-bit sum");
__global__ void __launch_bounds__(256) k_run_list(const unsigned *__restrict__ B, LD d, unsigned want, int *list, unsigned *wlist,
                                                  unsigned *nlist, unsigned *nwlist, const unsigned *__restrict__ skip) {
    grid_wait();
    __shared__ unsigned wsum[8], base, wbase;
    const unsigned off = skip ? __ldg(skip) : 0u;   // looked at late: no wait for it at the start
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    for (unsigned i0 = blockIdx.x * 256 * LIST_K; i0 < d.nwords; i0 += gridDim.x * 256 * LIST_K) {
        unsigned st[LIST_K], n = 0, any = 0;   // n: run starts | words << 16
#pragma unroll
        for (int k = 0; k < LIST_K; k++) {
            const unsigned i = i0 + (unsigned)(k * 256 + tid);
            st[k] = 0u;
            if (i < d.nwords) {
                const unsigned r = i / d.W, w = i - r * d.W;
                const unsigned c = class_word(B, d, r, w, want), pc = w ? class_word(B, d, r, w - 1, want) : 0u;
                st[k] = c & ~((c << 1) | (pc >> 31));
                any |= (c ? 1u : 0u) << k;
            }
            n += __popc(st[k]);
        }
        n += __popc(any) << 16;
        unsigned incl = n;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned t = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane == 31) wsum[wid] = incl;
        if (off) return;   // empty lists: nothing to do for the kernels that follow
        __syncthreads();
        if (tid == 0) {
            unsigned t = 0;
            for (int k = 0; k < 8; k++) t += wsum[k];
            if (t) {
                base = atomicAdd(nlist, t & 0xffffu);
                wbase = atomicAdd(nwlist, t >> 16);
            }
        }
        __syncthreads();
        unsigned before = incl - n;
        for (int k = 0; k < wid; k++) before += wsum[k];
        unsigned at = base + (before & 0xffffu), wat = wbase + (before >> 16);
#pragma unroll
        for (int k = 0; k < LIST_K; k++) {
            const unsigned i = i0 + (unsigned)(k * 256 + tid), r = i / d.W;
            const int x0 = (int)((long long)r * d.nx + (long long)(i - r * d.W) * 32);
            for (unsigned m = st[k]; m; m &= m - 1) list[at++] = x0 + __ffs(m) - 1;
            if (any >> k & 1u) wlist[wat++] = i;
        }
        __syncthreads();   // wsum and the bases are reused
    }
}

// the word holding run start s and the run's piece of it
__device__ __forceinline__ Word start_word(const unsigned *__restrict__ B, const LD &d, unsigned want, int s, unsigned &piece) {
    const unsigned r = (unsigned)s / (unsigned)d.nx, x = (unsigned)s - r * (unsigned)d.nx;
    const Word q = load_word(B, d, r, x >> 5, want);
    piece = piece_at(q.c, (int)(x & 31u));
    return q;
}

// Every run start of the class links to one run before it that it touches (itself
// if its first word touches none): a forest over all runs, without an atomic, whose
// trees are nearly the components.  z8 (may be null) is zeroed at the run starts (the
// edge flags the roots will carry), len (may be null) takes the run's length.
template <int NNB>
__global__ void __launch_bounds__(256) k_run_hook(const unsigned *__restrict__ B, LD d, unsigned want, const int *__restrict__ cs,
                                                  const int *__restrict__ list, const unsigned *__restrict__ nlist, int *L,
                                                  unsigned char *z8, unsigned *len) {
    grid_wait();
    const unsigned n = *nlist;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i];
        unsigned piece;
        Around<NNB> A;
        A.load(B, d, want, start_word(B, d, want, s, piece));
        int parent = s;
        bool found = false;
#pragma unroll
        for (int q = 0; q < ndirs(NNB); q++) {   // the first direction with a contact wins
            const unsigned t = piece & A.q[dir_k(q)].shifted(dir_x(q));
            if (!found && t) {
                found = true;
                parent = A.q[dir_k(q)].run(d, cs, __ffs(t) - 1 + dir_x(q));
            }
        }
        L[s] = parent;
        if (z8) z8[s] = 0;
        if (len) {
            Word q = A.q[0];
            unsigned l = __popc(piece);
            while ((piece >> 31) && (q.nc & 1u)) {
                q = load_word(B, d, q.r, q.w + 1, want);
                piece = piece_at(q.c, 0);
                l += __popc(piece);
            }
            len[s] = l;
        }
    }
}

// Every run start points at its root (links only ever move to ancestors, which come
// before them in raster order, so every walk ends).  The way found so far is left for
// the others every JUMPS links: they run in raster order more or less, and later
// walks are a few links long.
constexpr int JUMPS = 4;
__global__ void __launch_bounds__(256) k_run_jump(const int *__restrict__ list, const unsigned *__restrict__ nlist, int *L) {
    grid_wait();
    const unsigned n = *nlist;
    volatile int *V = L;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i];
        int p = V[s], at = p;
        for (bool more = true; more;) {
#pragma unroll
            for (int h = 0; h < JUMPS; h++) {
                const int q = V[p];
                more = q != p;
                p = q;
                if (!more) break;
            }
            if (p != at) V[s] = at = p;
        }
    }
}

// Union of the runs of the class with those of the rows before them: rows
// (y-1, z) and (y, z-1) for 6-connectivity, with x offsets -1..1 for 18 and
// rows (y-1, z-1), (y+1, z-1) for 18 (x offset 0) and 26 (-1..1).  A contact
// of voxel x with voxel x+dx of row k counts only if voxels x-1 and x+dx-1
// do not also touch: one union per overlap of two runs.  After the hooks and
// jumps nearly every contact joins runs with the same link already: the links of all
// directions' contacts are read together, and only different ones are united.
// A thread per word of the class (a thread per run walked long runs word by word: the
// background of the 512^3 CT volume took twice as long).
template <int NNB>
__global__ void __launch_bounds__(256) k_run_merge(const unsigned *__restrict__ B, LD d, unsigned want, const int *__restrict__ cs,
                                                   const unsigned *__restrict__ wlist, const unsigned *__restrict__ nwlist, int *L) {
    grid_wait();
    constexpr int ND = ndirs(NNB);
    const unsigned n = *nwlist;
    for (unsigned j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const unsigned i = wlist[j], r = i / d.W;
        const Word own = load_word(B, d, r, i - r * d.W, want);
        Around<NNB> A;
        A.load(B, d, want, own);
        const unsigned left = own.shifted(-1);
        unsigned m[ND], any = 0u;
#pragma unroll
        for (int k = 0; k < ND; k++) {
            const Word &q = A.q[dir_k(k)];
            m[k] = own.c & q.shifted(dir_x(k)) & ~(left & q.shifted(dir_x(k) - 1));
            any |= m[k];
        }
        while (any) {
            int a[ND], b[ND];
            any = 0u;
#pragma unroll
            for (int k = 0; k < ND; k++) {
                a[k] = b[k] = 0;
                if (m[k]) {
                    const int x = __ffs(m[k]) - 1;
                    a[k] = L[own.run(d, cs, x)];
                    b[k] = L[A.q[dir_k(k)].run(d, cs, x + dir_x(k))];
                    m[k] &= m[k] - 1u;
                    any |= m[k];
                }
            }
#pragma unroll
            for (int k = 0; k < ND; k++)
                if (a[k] != b[k]) unite(L, a[k], b[k]);
        }
    }
}

// every run start of the class points at its root; roots are counted.  The
// root search only reads: the one store of this kernel is a start's final
// root (a path-halving store could overwrite a root another thread has just
// stored with a lower ancestor).
__global__ void __launch_bounds__(256) k_run_flatten(const int *__restrict__ list, const unsigned *__restrict__ nlist, int *L,
                                                     unsigned *nroots) {
    grid_wait();
    const unsigned n = *nlist;
    unsigned cnt = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i], root = find_root(L, s);
        if (root == s) cnt++;
        else L[s] = root;
    }
    __shared__ unsigned all;   // one atomic per block: a few ns each on the one address, 13 us by warps
    if (threadIdx.x == 0) all = 0;
    __syncthreads();
    cnt = __reduce_add_sync(FULL, cnt);
    if ((threadIdx.x & 31) == 0 && cnt) atomicAdd(&all, cnt);
    __syncthreads();
    if (threadIdx.x == 0 && all) atomicAdd(nroots, all);
}

// Background components touching a face of the volume flag their root:
// items [0, nrows) take the runs holding x = 0 and x = nx-1 of a row, the items
// after them one word each of the rows on a y or z face (every run in it).  A
// flag is stored only if it is not set yet (most items name the same root).
__global__ void k_run_edges(const unsigned *__restrict__ B, LD d, const int *__restrict__ L, unsigned char *edge,
                            const unsigned *__restrict__ skip) {
    grid_wait();
    const unsigned off = skip ? __ldg(skip) : 0u;   // then no run has a link
    const unsigned nzf = d.nz > 1 ? 2u : 1u, nyf = d.ny > 1 ? 2u : 1u;
    const unsigned zrows = nzf * (unsigned)d.ny, yrows = d.nz > 2 ? nyf * (unsigned)(d.nz - 2) : 0u;
    const unsigned total = d.nrows + (zrows + yrows) * d.W;
    auto mark = [&](long long j) {
        const int root = L[j];
        if (!off && !edge[root]) edge[root] = 1;
    };
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        if (t < d.nrows) {
            const unsigned r = t;
            const long long base = (long long)r * d.nx;
            if (class_word(B, d, r, 0, 0u) & 1u) mark(base);
            unsigned w = d.W - 1;
            int b = (d.nx - 1) & 31;
            unsigned c = class_word(B, d, r, w, 0u);
            if (!((c >> b) & 1u)) continue;
            for (;;) {   // back to the run's start (x = 0 of a background run is one)
                const unsigned pc = w ? class_word(B, d, r, w - 1, 0u) : 0u;
                const int ls = last_start(c & ~((c << 1) | (pc >> 31)), (int)w * 32, b);
                if (ls >= 0) {
                    mark(base + ls);
                    break;
                }
                w--;
                b = 31;
                c = pc;
            }
            continue;
        }
        const unsigned u = t - d.nrows, fr = u / d.W, w = u - fr * d.W;
        unsigned r;
        if (fr < zrows) {   // slices z = 0 and z = nz-1
            const unsigned side = fr / (unsigned)d.ny, y = fr - side * (unsigned)d.ny;
            r = (side ? (unsigned)(d.nz - 1) * (unsigned)d.ny : 0u) + y;
        } else {            // rows y = 0 and y = ny-1 of the slices between
            const unsigned v = fr - zrows, side = v / (unsigned)(d.nz - 2), z = 1 + v - side * (unsigned)(d.nz - 2);
            r = z * (unsigned)d.ny + (side ? (unsigned)(d.ny - 1) : 0u);
        }
        const unsigned c = class_word(B, d, r, w, 0u), pc = w ? class_word(B, d, r, w - 1, 0u) : 0u;
        const long long base = (long long)r * d.nx + (long long)w * 32;
        for (unsigned st = c & ~((c << 1) | (pc >> 31)); st; st &= st - 1) mark(base + __ffs(st) - 1);
    }
}

// sets the bits of the run that starts at s in out
__device__ __forceinline__ void put_run(const unsigned *__restrict__ B, const LD &d, unsigned want, int s, unsigned *out) {
    unsigned piece;
    for (Word q = start_word(B, d, want, s, piece);;) {
        atomicOr(out + (size_t)q.r * d.W + q.w, piece);
        if (!(piece >> 31) || !(q.nc & 1u)) break;
        q = load_word(B, d, q.r, q.w + 1, want);
        piece = piece_at(q.c, 0);
    }
}

// bubbles (background components away from every face) become foreground,
// only when the background has at least two components (src/bwlabel.c:488-491);
// out: the foreground, a copy (the background's words must stay what they were)
__global__ void __launch_bounds__(256) k_run_fill(const unsigned *__restrict__ B, LD d, const int *__restrict__ list,
                                                  const unsigned *__restrict__ nlist, const int *__restrict__ L,
                                                  const unsigned char *__restrict__ edge, const unsigned *__restrict__ nbg,
                                                  unsigned *out) {
    grid_wait();
    if (*nbg <= 1) return;
    const unsigned n = *nlist;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i];
        if (!edge[L[s]]) put_run(B, d, 0u, s, out);
    }
}

// Component sizes, from the runs' lengths (k_run_hook): every run that is no root adds
// its own to its root's.  Most runs belong to a few large components, so a lane keeps the
// heaviest root it meets to itself, and the block adds up what belongs to the
// heaviest root of its first lane (an atomic per warp and root, roots included, with the run walked
// again took 91 us for an int16 scan's million runs, 48 now).
__global__ void __launch_bounds__(256) k_run_sizes(const int *__restrict__ list, const unsigned *__restrict__ nlist,
                                                   const int *__restrict__ L, unsigned *cnt) {
    grid_wait();
    __shared__ int hot;
    __shared__ unsigned total;
    const unsigned n = *nlist;
    int mine = -1;
    unsigned sum = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i], root = L[s];
        if (root == s) continue;
        const unsigned len = cnt[s];   // only roots' change
        if (root == mine) {
            sum += len;
        } else if (len <= sum) {
            atomicAdd(&cnt[root], len);
        } else {
            if (sum) atomicAdd(&cnt[mine], sum);
            mine = root;
            sum = len;
        }
    }
    if (threadIdx.x == 0) {
        hot = mine;
        total = 0;
    }
    __syncthreads();
    const unsigned w = __reduce_add_sync(FULL, mine == hot ? sum : 0u);
    if ((threadIdx.x & 31) == 0 && w) atomicAdd(&total, w);
    if (mine != hot && sum) atomicAdd(&cnt[mine], sum);
    __syncthreads();
    if (threadIdx.x == 0 && total) atomicAdd(&cnt[hot], total);
}

// largest component; ties go to the smallest root (first in raster order)
__global__ void __launch_bounds__(256) k_run_best(const int *__restrict__ list, const unsigned *__restrict__ nlist,
                                                  const int *__restrict__ L, const unsigned *__restrict__ cnt,
                                                  unsigned long long *best) {
    grid_wait();
    const unsigned n = *nlist;
    unsigned long long b = 0;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i];
        if (L[s] != s) continue;
        const unsigned long long k = ((unsigned long long)cnt[s] << 32) | (0xffffffffu - (unsigned)s);
        b = k > b ? k : b;
    }
    for (int o = 16; o; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(FULL, b, o);
        b = t > b ? t : b;
    }
    __shared__ unsigned long long all;   // one atomic per block, and only while it changes something
    if (threadIdx.x == 0) all = 0;
    __syncthreads();
    if ((threadIdx.x & 31) == 0 && b) atomicMax(&all, b);
    __syncthreads();
    if (threadIdx.x == 0 && all > *(volatile unsigned long long *)best) atomicMax(best, all);
}

// bits of the voxels of the largest component (K cleared before)
__global__ void __launch_bounds__(256) k_run_keep(const unsigned *__restrict__ B, LD d, const int *__restrict__ list,
                                                  const unsigned *__restrict__ nlist, const int *__restrict__ L,
                                                  const unsigned long long *__restrict__ best, unsigned *K) {
    grid_wait();
    const unsigned long long bk = *best;
    if (!bk) return;
    const int root = (int)(0xffffffffu - (unsigned)(bk & 0xffffffffu));
    const unsigned n = *nlist;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int s = list[i];
        if (L[s] == root) put_run(B, d, 1u, s, K);
    }
}

__global__ void k_nl_from(const unsigned *nroots, bool only_largest, int *nl) {
    grid_wait();
    *nl = only_largest ? (*nroots > 0 ? 1 : 0) : (int)*nroots;
}

// The labelled volume (src/meshify.c:330-342) without writing it.  Kept voxels (K) are
// at or above iso (raised to it when filled); a voxel neither kept nor in the dilation of the
// kept set (the 26-neighbourhood without (-1,-1,-1), interior voxels only;
// src/meshify.c:218-264) is the minimum mn, below iso; only the voxels of the
// dilation's shell keep their values, and only those are read here.  Leaves the sign
// bitmap of the result (S: value - iso > -FLT_EPSILON, or value >= iso for
// at_or_above; mn must be on the other side), the kept or dilated voxels (KD), and in
// *st the bbox of the voxels >= iso and the count of masked ones.  Marching cubes reads
// values next to sign changes only; they are put right there (lab_apply,
// smooth.cu: k_od_post).  512^3: 203 us when every voxel was written.
// With R3 = K(x-1) | K(x) | K(x+1) and R2 = K(x) | K(x+1) of a row, the dilation is R3
// of rows y-1..y+1 in slices z and z+1, R3 of rows y and y+1 in slice z-1, and R2 of
// row y-1 in slice z-1.  A lane per word, 32 consecutive words per warp.
__global__ void __launch_bounds__(256) k_lab_shell(const unsigned *__restrict__ K, LD d, const float *__restrict__ vol, float iso,
                                                   bool at_or_above, unsigned *S, unsigned *KD, VolStats *st) {
    grid_wait();
    smooth::Acc acc;
    acc.init();
    unsigned masked = 0;
    const int lane = threadIdx.x & 31;
    // rows used: 0..2 = y-1..y+1 in slice z, 3..5 in slice z+1, 6 = (y, z-1), 7 = (y+1, z-1), 8 = (y-1, z-1)
    constexpr int DY[9] = {-1, 0, 1, -1, 0, 1, 0, 1, -1}, DZ[9] = {0, 0, 0, 1, 1, 1, -1, -1, -1};
    const unsigned n32 = (d.nwords + 31u) & ~31u, slice = d.W * (unsigned)d.ny;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n32; i += gridDim.x * blockDim.x) {   // whole warps
        const bool live = i < d.nwords;
        const unsigned r = live ? i / d.W : 0u, w = live ? i - r * d.W : 0u;
        const int z = (int)(r / (unsigned)d.ny), y = (int)(r - (unsigned)z * (unsigned)d.ny);
        const unsigned valid = live ? valid_bits(d, w) : 0u;
        unsigned on = 0u, kept = 0u;
#pragma unroll
        for (int k = 0; k < 9; k++) {
            const int yy = y + DY[k], zz = z + DZ[k];
            const bool in = live && yy >= 0 && zz >= 0 && yy < d.ny && zz < d.nz;
            const unsigned q = in ? i + (unsigned)(DZ[k] * (int)slice + DY[k] * (int)d.W) : 0u;
            const unsigned cur = in ? __ldg(K + q) : 0u;
            unsigned prv = __shfl_up_sync(FULL, cur, 1), nxt = __shfl_down_sync(FULL, cur, 1);
            if (lane == 0) prv = in && w ? __ldg(K + q - 1) : 0u;
            if (lane == 31) nxt = in && w + 1 < d.W ? __ldg(K + q + 1) : 0u;
            if (w == 0) prv = 0u;
            if (w + 1 >= d.W) nxt = 0u;
            on |= cur | (cur >> 1) | (nxt << 31) | (k < 8 ? (cur << 1) | (prv >> 31) : 0u);   // row 8: no K(x-1)
            if (k == 1) kept = cur;
        }
        // interior voxels only
        if (y > 0 && z > 0 && y < d.ny - 1 && z < d.nz - 1) {
            if (w == 0) on &= ~1u;
            if ((int)w * 32 + 31 >= d.nx - 1) on &= (int)w * 32 < d.nx - 1 ? (1u << (d.nx - 1 - (int)w * 32)) - 1u : 0u;
        } else {
            on = 0u;
        }
        const unsigned shell = on & ~kept & valid, kd = kept | shell;
        masked += __popc(valid & ~kd);
        unsigned sg = kept, ge = kept;
        const long long base = (long long)r * d.nx + (long long)w * 32;
        for (unsigned busy = __ballot_sync(FULL, shell != 0u); busy;) {   // the shell's values, four words in flight
            int j[4];
            float v[4];
            unsigned sj[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                j[u] = busy ? __ffs(busy) - 1 : -1;
                busy &= busy - 1u;
                sj[u] = __shfl_sync(FULL, shell, j[u] & 31);
                const long long bj = __shfl_sync(FULL, base, j[u] & 31);
                v[u] = j[u] >= 0 && (sj[u] >> lane & 1u) ? __ldg(vol + bj + lane) : 0.f;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const bool in = j[u] >= 0 && (sj[u] >> lane & 1u);
                const unsigned a = __ballot_sync(FULL, in && v[u] >= iso), p = __ballot_sync(FULL, in && __fsub_rn(v[u], iso) > -N2M_FLT_EPS);
                if (lane == j[u]) {
                    ge |= a;
                    sg |= at_or_above ? a : p;
                }
            }
        }
        if (live) {
            S[i] = sg;
            KD[i] = kd;
        }
        if (ge) {
            acc.lo0 = min(acc.lo0, (int)w * 32 + __ffs(ge) - 1); acc.hi0 = max(acc.hi0, (int)w * 32 + 31 - __clz(ge));
            acc.lo1 = min(acc.lo1, y); acc.hi1 = max(acc.hi1, y);
            acc.lo2 = min(acc.lo2, z); acc.hi2 = max(acc.hi2, z);
        }
    }
    masked = __reduce_add_sync(FULL, masked);
    if (lane == 0 && masked) atomicAdd(&st->masked, masked);
    acc.flush(st, false);
}

// the labelling's effect on the values marching cubes will read: the marked voxels of `need`
__global__ void __launch_bounds__(256) k_lab_apply(const unsigned *__restrict__ need, LD d, LabelPost P, float *vol) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    const unsigned n32 = (d.nwords + 31u) & ~31u;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n32; i += gridDim.x * blockDim.x) {   // whole warps
        const unsigned m = i < d.nwords ? need[i] : 0u, r = i / d.W;
        unsigned kept = 0u, kd = 0u;
        if (m) {
            kept = P.K[i];
            kd = P.KD[i];
        }
        const long long base = (long long)r * d.nx + (long long)(i - r * d.W) * 32;
        for (unsigned busy = __ballot_sync(FULL, m != 0u); busy; busy &= busy - 1u) {
            const int k = __ffs(busy) - 1;
            const unsigned mk = __shfl_sync(FULL, m, k), kk = __shfl_sync(FULL, kept, k), dk = __shfl_sync(FULL, kd, k);
            float *v = vol + __shfl_sync(FULL, base, k) + lane;
            if (!(mk >> lane & 1u)) continue;
            if (!(dk >> lane & 1u)) *v = P.mn;
            else if (P.fill && (kk >> lane & 1u)) *v = fmaxf(*v, P.iso);
        }
    }
}

// The labelled volume written out (without -l 1, or when nothing is masked out and its
// minimum has to be found), one warp per row, 32 voxels a word, with the range and
// bbox of the result.  Kept voxels (K) are raised to iso when FILL; with
// LARGEST, voxels neither kept nor in the dilation of the kept set (the
// 26-neighbourhood without (-1,-1,-1), interior voxels only;
// src/meshify.c:218-264) become mn and are not read.  With R3 = K(x-1) | K(x) |
// K(x+1) and R2 = K(x) | K(x+1) of a row, the dilation is R3 of rows y-1..y+1
// in slices z and z+1, R3 of rows y and y+1 in slice z-1, and R2 of row y-1 in
// slice z-1.  The keep words of a row are loaded 32 at a time (lane l holds
// word c0 + l) and broadcast; 32 words with no kept voxel within reach are
// written without being read.
template <bool LARGEST, bool FILL, bool ONE>   // ONE: rows of at most 32 words
__global__ void __launch_bounds__(256) k_lab_final(const unsigned *__restrict__ K, LD d, float *vol, float iso, float mn,
                                                   VolStats *st, bool vec4) {
    grid_wait();
    smooth::Acc acc;
    acc.init();
    unsigned masked = 0;
    const int lane = threadIdx.x & 31;
    // rows used: 0..2 = y-1..y+1 in slice z, 3..5 in slice z+1, 6 = (y, z-1), 7 = (y+1, z-1), 8 = (y-1, z-1)
    const int DY[9] = {-1, 0, 1, -1, 0, 1, 0, 1, -1}, DZ[9] = {0, 0, 0, 1, 1, 1, -1, -1, -1};
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < d.nrows; r += (gridDim.x * blockDim.x) >> 5) {
        const int z = (int)(r / (unsigned)d.ny), y = (int)(r - (unsigned)z * (unsigned)d.ny);
        float *row = vol + (long long)r * d.nx;
        if (!LARGEST) {
            const unsigned *K0 = K + (size_t)r * d.W;
            for (unsigned c0 = 0; c0 < d.W; c0 += 32) {
                const unsigned kk = c0 + lane < d.W ? K0[c0 + lane] : 0u;
                const unsigned wend = min(d.W, c0 + 32);
#pragma unroll 4
                for (unsigned w = c0; w < wend; w++) {
                    const unsigned kw = __shfl_sync(FULL, kk, (int)(w - c0));
                    const int x = (int)w * 32 + lane;
                    if (x >= d.nx) continue;
                    float v = row[x];
                    if (FILL && ((kw >> lane) & 1u)) {
                        v = fmaxf(v, iso);
                        row[x] = v;
                    }
                    acc.add(v, x, y, z, iso);
                }
            }
            continue;
        }
        const bool ryz = y > 0 && z > 0 && y < d.ny - 1 && z < d.nz - 1;
        unsigned carry[9];   // word c0 - 1 of each row
#pragma unroll
        for (int k = 0; k < 9; k++) carry[k] = 0u;
        for (unsigned c0 = 0; c0 < d.W; c0 += 32) {
            // lane l: word c0 + l of the kept set and of its dilation (the row's own word for
            // `kept`); the words next to it come from the neighbouring lanes
            unsigned on = 0u, kept = 0u;
#pragma unroll
            for (int k = 0; k < 9; k++) {
                const int yy = y + DY[k], zz = z + DZ[k];
                const bool in = yy >= 0 && zz >= 0 && yy < d.ny && zz < d.nz;
                const unsigned *Kk = K + ((size_t)(in ? zz : 0) * d.ny + (in ? yy : 0)) * d.W;
                const unsigned cur = in && c0 + lane < d.W ? Kk[c0 + lane] : 0u;
                unsigned prv = __shfl_up_sync(FULL, cur, 1), nxt = __shfl_down_sync(FULL, cur, 1);
                if (lane == 0) prv = carry[k];
                if (lane == 31) nxt = !ONE && in && c0 + 32 < d.W ? Kk[c0 + 32] : 0u;
                if (!ONE) carry[k] = __shfl_sync(FULL, cur, 31);
                on |= cur | (cur >> 1) | (nxt << 31) | (k < 8 ? (cur << 1) | (prv >> 31) : 0u);   // row 8: no K(x-1)
                if (k == 1) kept = cur;
            }
            const unsigned wend = min(d.W, c0 + 32);
            if (!__any_sync(FULL, on != 0u)) {   // nothing kept within reach: all mn
                const int xb = (int)c0 * 32, xe = min(d.nx, (int)wend * 32);
                if (vec4) {   // rows of a multiple of 4 voxels on 16-byte boundaries
                    float4 *r4 = (float4 *)(row + xb);
                    for (int q = lane; q < (xe - xb) >> 2; q += 32) {
                        r4[q] = make_float4(mn, mn, mn, mn);
                        masked += 4;
                    }
                } else {
                    for (int x = xb + lane; x < xe; x += 32) {
                        row[x] = mn;
                        masked++;
                    }
                }
                acc.mn = fminf(acc.mn, mn);
                acc.mx = fmaxf(acc.mx, mn);
                continue;
            }
            for (unsigned w = c0; w < wend; w++) {
                const unsigned onw = __shfl_sync(FULL, on, (int)(w - c0)), kw = __shfl_sync(FULL, kept, (int)(w - c0));
                const int x = (int)w * 32 + lane;
                if (x >= d.nx) continue;
                const bool kp = (kw >> lane) & 1u;
                const bool interior = ryz && x > 0 && x < d.nx - 1;
                float v;
                if (!(kp || (interior && ((onw >> lane) & 1u)))) {
                    v = mn;
                    row[x] = v;
                    masked++;
                } else {
                    v = row[x];
                    if (FILL && kp) {
                        v = fmaxf(v, iso);
                        row[x] = v;
                    }
                }
                acc.add(v, x, y, z, iso);
            }
        }
    }
    for (int o = 16; o; o >>= 1) masked += __shfl_xor_sync(FULL, masked, o);
    if (lane == 0 && masked) atomicAdd(&st->masked, masked);
    acc.flush(st, true);
}

// bwlabel() output: 0/1 of the kept set
__global__ void __launch_bounds__(256) k_write_keep(const unsigned *__restrict__ K, LD d, float *vol) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < d.nrows; r += (gridDim.x * blockDim.x) >> 5) {
        float *row = vol + (long long)r * d.nx;
        for (unsigned w = 0; w < d.W; w++) {
            const unsigned kw = K[(size_t)r * d.W + w];
            const int x = (int)w * 32 + lane;
            if (x < d.nx) row[x] = (kw >> lane) & 1u ? 1.0f : 0.0f;
        }
    }
}

// bwlabel() labels: 1 + rank of the component's root among the roots in
// raster order.  Roots per word, then (after a scan) each root's rank.
__global__ void k_root_count(const unsigned *__restrict__ B, LD d, const int *__restrict__ L, unsigned *rc) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < d.nwords; i += gridDim.x * blockDim.x) {
        const unsigned r = i / d.W, w = i - r * d.W;
        const unsigned c = class_word(B, d, r, w, 1u), pc = w ? class_word(B, d, r, w - 1, 1u) : 0u;
        const long long base = (long long)r * d.nx + (long long)w * 32;
        unsigned n = 0;
        for (unsigned st = c & ~((c << 1) | (pc >> 31)); st; st &= st - 1) {
            const int s = (int)(base + __ffs(st) - 1);
            n += L[s] == s;
        }
        rc[i] = n;
    }
}

__global__ void k_root_rank(const unsigned *__restrict__ B, LD d, const int *__restrict__ L,
                            const unsigned *__restrict__ rc, unsigned *rank) {
    grid_wait();
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < d.nwords; i += gridDim.x * blockDim.x) {
        const unsigned r = i / d.W, w = i - r * d.W;
        const unsigned c = class_word(B, d, r, w, 1u), pc = w ? class_word(B, d, r, w - 1, 1u) : 0u;
        const long long base = (long long)r * d.nx + (long long)w * 32;
        unsigned k = rc[i];
        for (unsigned st = c & ~((c << 1) | (pc >> 31)); st; st &= st - 1) {
            const int s = (int)(base + __ffs(st) - 1);
            if (L[s] == s) rank[s] = k++;
        }
    }
}

__global__ void __launch_bounds__(256) k_write_labels(const unsigned *__restrict__ B, LD d, const int *__restrict__ L,
                                                      const unsigned *__restrict__ rank, float *vol) {
    grid_wait();
    const int lane = threadIdx.x & 31;
    for (unsigned r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < d.nrows; r += (gridDim.x * blockDim.x) >> 5) {
        float *row = vol + (long long)r * d.nx;
        const long long base = (long long)r * d.nx;
        int carry = -1;   // last run start of the words before
        unsigned pc = 0;
        for (unsigned w = 0; w < d.W; w++) {
            const unsigned c = B[(size_t)r * d.W + w];
            const unsigned starts = c & ~((c << 1) | (pc >> 31));
            const int x0 = (int)w * 32, x = x0 + lane;
            if (x < d.nx) {
                float v = 0.0f;
                if ((c >> lane) & 1u) {
                    const int s0 = last_start(starts, x0, lane);
                    v = (float)(rank[L[base + (s0 >= 0 ? s0 : carry)]] + 1u);
                }
                row[x] = v;
            }
            if (starts) carry = x0 + 31 - __clz(starts);
            pc = c;
        }
    }
}

inline unsigned gsz(long long n) {
    long long b = (n + 255) / 256;
    if (b > 152 * 64) b = 152 * 64;
    return b ? (unsigned)b : 1u;
}
// row kernels: one warp per 32/seg rows
inline unsigned rgrid(const LD &d) {
    const long long warps = ((long long)d.nrows * d.seg + 31) / 32;
    return (unsigned)std::max<long long>(1, std::min<long long>((warps + 7) / 8, 152 * 16));
}
// one warp per row
inline unsigned wgrid(const LD &d) {
    return (unsigned)std::max<long long>(1, std::min<long long>(((long long)d.nrows + 7) / 8, 152 * 16));
}

LD make_ld(int nx, int ny, int nz) {
    LD d;
    d.nx = nx; d.ny = ny; d.nz = nz;
    d.nxy = (long long)nx * ny;
    d.n = d.nxy * nz;
    d.W = (unsigned)(nx + 31) / 32;
    d.nrows = (unsigned)ny * (unsigned)nz;
    d.nwords = d.W * d.nrows;
    d.seg = 1;
    while (d.seg < 32 && (unsigned)d.seg < d.W) d.seg <<= 1;
    return d;
}

// a thread per run, all resident at once
inline unsigned run_grid(const LD &d) { return std::min(gsz(d.nwords), 152u * 8u); }

struct Misc {
    unsigned nbg, nfg;
    unsigned long long best;
    int nl;
    unsigned nlist[2], nwlist[2];   // run starts and words of the background and the foreground
};

n2m_status components(LabelWork &w, const LD &d, const unsigned *B, unsigned want, int conn, Misc *misc, unsigned char *z8,
                      unsigned *z32, const unsigned *skip, cudaStream_t s) {
    int *L = w.lab.as<int>(), *list = w.list.as<int>();
    unsigned *nlist = &misc->nlist[want];
    int *cs = w.cs.as<int>();
    const unsigned lg = std::max(1u, std::min((d.nwords + 256 * LIST_K - 1) / (256 * LIST_K), 152u * 16u));
    const unsigned g = run_grid(d), wg = gsz(d.nwords);
    unsigned *wlist = w.wlist.as<unsigned>(), *nwlist = &misc->nwlist[want];
    n2m_launch(k_run_starts, rgrid(d), 256, 0, s, B, d, want, cs);
    n2m_launch(k_run_list, lg, 256, 0, s, B, d, want, list, wlist, nlist, nwlist, skip);
    if (conn == 6) n2m_launch(k_run_hook<3>, 2 * g, 128, 0, s, B, d, want, cs, list, nlist, L, z8, z32);
    else if (conn == 18) n2m_launch(k_run_hook<9>, 2 * g, 128, 0, s, B, d, want, cs, list, nlist, L, z8, z32);
    else n2m_launch(k_run_hook<13>, 2 * g, 128, 0, s, B, d, want, cs, list, nlist, L, z8, z32);
    // once every start points at its tree's root, nearly every contact of the merge joins equal links
    n2m_launch(k_run_jump, 2 * g, 128, 0, s, list, nlist, L);
    if (conn == 6) n2m_launch(k_run_merge<3>, 4 * wg, 64, 0, s, B, d, want, cs, wlist, nwlist, L);
    else if (conn == 18) n2m_launch(k_run_merge<9>, 4 * wg, 64, 0, s, B, d, want, cs, wlist, nwlist, L);
    else n2m_launch(k_run_merge<13>, 4 * wg, 64, 0, s, B, d, want, cs, wlist, nwlist, L);
    n2m_launch(k_run_flatten, 2 * g, 128, 0, s, list, nlist, L, want ? &misc->nfg : &misc->nbg);
    CKL();
    return N2M_OK;
}

// the class bits in w.mask on entry; *keep: the kept voxels' bits on return
// (the foreground after filling, or its largest component); skip: see run_labelling
n2m_status label_core(LabelWork &w, const LD &d, int conn, bool only_largest, bool fill_bubbles, const unsigned *skip,
                      cudaStream_t s, const unsigned **keep) {
    CKS(w.lab.ensure((size_t)d.n * sizeof(int)));
    CKS(w.list.ensure(((size_t)d.nrows * ((d.nx + 1) / 2)) * sizeof(int)));   // every second voxel of a row at most
    CKS(w.wlist.ensure((size_t)d.nwords * sizeof(unsigned)));
    CKS(w.misc.ensure(sizeof(Misc)));
    Misc *misc = w.misc.as<Misc>();
    CK(cudaMemsetAsync(misc, 0, sizeof(Misc), s));
    const unsigned *B = w.mask.as<unsigned>();
    CKS(w.cs.ensure((size_t)d.nwords * sizeof(int)));
    if (fill_bubbles) {
        CKS(w.edge.ensure((size_t)d.n));
        CKS(w.filled.ensure((size_t)d.nwords * sizeof(unsigned)));
        CKS(components(w, d, B, 0u, 6, misc, w.edge.as<unsigned char>(), nullptr, skip, s));
        n2m_launch(k_run_edges, gsz((long long)d.nrows + 4ll * (d.nx + d.ny + d.nz) * d.W), 256, 0, s, B, d, w.lab.as<int>(),
                   w.edge.as<unsigned char>(), skip);
        CK(cudaMemcpyAsync(w.filled.p, B, (size_t)d.nwords * sizeof(unsigned), cudaMemcpyDeviceToDevice, s));
        n2m_launch(k_run_fill, run_grid(d), 256, 0, s, B, d, w.list.as<int>(), &misc->nlist[0], w.lab.as<int>(),
                   w.edge.as<unsigned char>(), &misc->nbg, w.filled.as<unsigned>());
        CKL();
        B = w.filled.as<unsigned>();
    }
    if (only_largest) CKS(w.cnt.ensure((size_t)d.n * sizeof(unsigned)));
    CKS(components(w, d, B, 1u, conn, misc, nullptr, only_largest ? w.cnt.as<unsigned>() : nullptr, skip, s));
    *keep = B;
    if (only_largest) {
        CKS(w.keep.ensure((size_t)d.nwords * sizeof(unsigned)));
        CK(cudaMemsetAsync(w.keep.p, 0, (size_t)d.nwords * sizeof(unsigned), s));
        n2m_launch(k_run_sizes, run_grid(d), 256, 0, s, w.list.as<int>(), &misc->nlist[1], w.lab.as<int>(),
                   w.cnt.as<unsigned>());
        n2m_launch(k_run_best, run_grid(d), 256, 0, s, w.list.as<int>(), &misc->nlist[1], w.lab.as<int>(), w.cnt.as<unsigned>(),
                   &misc->best);
        n2m_launch(k_run_keep, run_grid(d), 256, 0, s, B, d, w.list.as<int>(), &misc->nlist[1], w.lab.as<int>(), &misc->best,
                   w.keep.as<unsigned>());
        *keep = w.keep.as<unsigned>();
    }
    n2m_launch(k_nl_from, 1, 1, 0, s, &misc->nfg, only_largest, &misc->nl);
    CKL();
    return N2M_OK;
}

n2m_status class_bits(LabelWork &w, const LD &d, const float *vol, float iso, bool nonzero, cudaStream_t s) {
    if (d.n > 0x7fffffffLL) {
        n2m_set_error("labelling supports at most 2^31-1 voxels");
        return N2M_ERR_TOO_LARGE;
    }
    CKS(w.mask.ensure((size_t)d.nwords * sizeof(unsigned)));
    n2m_launch(k_lab_bits, wgrid(d), 256, 0, s, vol, d, iso, nonzero, w.mask.as<unsigned>());
    CKL();
    return N2M_OK;
}
}  // namespace

n2m_status run_labelling(const float *vol, int nx, int ny, int nz, float iso, bool only_largest, bool fill_bubbles,
                         bool at_or_above, LabelWork &w, VolStats *st, cudaStream_t s, const unsigned *vsign, const unsigned *skip,
                         LabelPost *post) {
    const LD d = make_ld(nx, ny, nz);
    if (vsign) {
        if (d.n > 0x7fffffffLL) {
            n2m_set_error("labelling supports at most 2^31-1 voxels");
            return N2M_ERR_TOO_LARGE;
        }
        CKS(w.mask.ensure((size_t)d.nwords * sizeof(unsigned)));
        n2m_launch(k_lab_bits_vsign, gsz(d.nwords), 256, 0, s, vsign, d, (unsigned)(ny + 7) / 8, w.mask.as<unsigned>());
        CKL();
    } else {
        CKS(class_bits(w, d, vol, iso, false, s));
    }
    const unsigned *K;
    CKS(label_core(w, d, 18, only_largest, fill_bubbles, skip, s, &K));
    *post = LabelPost{K, nullptr, nullptr, d.W, 0.f, iso, fill_bubbles, only_largest};
    if (only_largest) {
        CKS(w.shell.ensure(2 * (size_t)d.nwords * sizeof(unsigned)));
        unsigned *S = w.shell.as<unsigned>(), *KD = S + d.nwords;
        n2m_launch(k_lab_shell, std::min(gsz(d.nwords), 152u * 16u), 256, 0, s, K, d, vol, iso, at_or_above, S, KD, st);
        CKL();
        post->S = S;
        post->KD = KD;
    }
    return N2M_OK;
}

n2m_status lab_write(float *vol, int nx, int ny, int nz, const LabelPost &P, VolStats *st, cudaStream_t s) {
    const LD d = make_ld(nx, ny, nz);
    const unsigned g = wgrid(d);
    const bool v4 = nx % 4 == 0 && ((uintptr_t)vol & 15) == 0, one = d.W <= 32;
    const unsigned *K = P.K;
    const float iso = P.iso, mn = P.mn;
    if (P.largest && P.fill && one) n2m_launch(k_lab_final<true, true, true>, g, 256, 0, s, K, d, vol, iso, mn, st,
                                               v4);
    else if (P.largest && P.fill) n2m_launch(k_lab_final<true, true, false>, g, 256, 0, s, K, d, vol, iso, mn, st,
                                             v4);
    else if (P.largest && one) n2m_launch(k_lab_final<true, false, true>, g, 256, 0, s, K, d, vol, iso, mn, st, v4);
    else if (P.largest) n2m_launch(k_lab_final<true, false, false>, g, 256, 0, s, K, d, vol, iso, mn, st, v4);
    else if (P.fill) n2m_launch(k_lab_final<false, true, false>, g, 256, 0, s, K, d, vol, iso, mn, st, v4);
    else n2m_launch(k_lab_final<false, false, false>, g, 256, 0, s, K, d, vol, iso, mn, st, v4);
    CKL();
    return N2M_OK;
}

n2m_status lab_apply(float *vol, int nx, int ny, int nz, const unsigned *need, const LabelPost &P, cudaStream_t s) {
    const LD d = make_ld(nx, ny, nz);
    n2m_launch(k_lab_apply, std::min(gsz(d.nwords), 152u * 16u), 256, 0, s, need, d, P, vol);
    CKL();
    return N2M_OK;
}

n2m_status run_bwlabel(float *vol, int nx, int ny, int nz, int conn, bool only_largest, bool fill_bubbles,
                       LabelWork &w, ScanWork &sw, int *d_nl, cudaStream_t s) {
    const LD d = make_ld(nx, ny, nz);
    CKS(class_bits(w, d, vol, 0.0f, true, s));
    const unsigned *K;
    CKS(label_core(w, d, conn, only_largest, fill_bubbles, nullptr, s, &K));
    if (only_largest) {
        n2m_launch(k_write_keep, wgrid(d), 256, 0, s, K, d, vol);
    } else {
        CKS(w.rc.ensure(((size_t)d.nwords + 1) * sizeof(unsigned)));
        CKS(w.cnt.ensure((size_t)d.n * sizeof(unsigned)));
        unsigned *rc = w.rc.as<unsigned>();
        CK(cudaMemsetAsync(rc + d.nwords, 0, sizeof(unsigned), s));
        n2m_launch(k_root_count, gsz(d.nwords), 256, 0, s, K, d, w.lab.as<int>(), rc);
        CKL();
        CKS(scan_u32(rc, (size_t)d.nwords + 1, rc + d.nwords, sw, s));
        n2m_launch(k_root_rank, gsz(d.nwords), 256, 0, s, K, d, w.lab.as<int>(), rc, w.cnt.as<unsigned>());
        n2m_launch(k_write_labels, wgrid(d), 256, 0, s, K, d, w.lab.as<int>(), w.cnt.as<unsigned>(), vol);
    }
    CK(cudaMemcpyAsync(d_nl, &w.misc.as<Misc>()->nl, sizeof(int), cudaMemcpyDeviceToDevice, s));
    CKL();
    return N2M_OK;
}
