// Descriptor matching on uint8 RootSIFT descriptors.
//
//   k_bf_exact    exhaustive nearest / second-nearest squared distance on the CUDA cores: exact
//                 32-bit integer distances (the plain path of matching._ratio_match_bf,
//                 app/planesite/matching.py:86-100)
//   k_bf_merge    merge of the per-split top-2, float32 ratio test, one-to-one keys
//   k_gb_*        prior-guided candidates within a radius on a uniform grid, exact integer
//                 distances (matching._guided, app/planesite/matching.py:113-152), one pair or a batch
//   k_unique      one match per target: atomicMin on (distance << 32 | query) keys
//                 (matching._unique, app/planesite/matching.py:103-110), then target-ordered
//                 compaction
//
// Exactness: descriptors are uint8 and every squared distance na + nb - 2 a.b is an integer below
// 2^24, so FP32 FMA accumulation in any order, integer dp4a, and BF16 x BF16 -> FP32 tensor-core
// products all give the same values as the reference's float32 BLAS. Results therefore depend only
// on the values and the tie rules, which follow the reference.
#include <cub/cub.cuh>

#include <atomic>
#include <mutex>

#include "fsb_internal.cuh"
#include "unique.cuh"

namespace fsb {
namespace {

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// ------------------------------------------------------------------------- dense tiles
constexpr int BN = 128;            // target rows per tile
constexpr int BF_PITCH = 144;      // bytes per staged row: rows 16 bytes apart mod 128, so the eight
                                   // rows of a quarter-warp's loads fall in different banks

struct Top2 {
    float b1, b2;
    int i1;
};

__device__ __forceinline__ void top2_push(Top2& t, float d, int j) {
    if (d < t.b1) {
        t.b2 = t.b1;
        t.b1 = d;
        t.i1 = j;
    } else if (d < t.b2) {
        t.b2 = d;
    }
}

__device__ __forceinline__ Top2 top2_merge(Top2 a, Top2 b) {
    Top2 r;
    if (a.b1 < b.b1 || (a.b1 == b.b1 && a.i1 <= b.i1)) {
        r.b1 = a.b1; r.i1 = a.i1; r.b2 = fminf(a.b2, b.b1);
    } else {
        r.b1 = b.b1; r.i1 = b.i1; r.b2 = fminf(b.b2, a.b1);
    }
    return r;
}

__device__ __forceinline__ void bf_cp_async(void* dst, const void* src, bool wide) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if (wide) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    } else {
#pragma unroll
        for (int k = 0; k < 16; k += 4)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + k), "l"((const char*)src + k) : "memory");
    }
}

// rows r0 .. r0 + ROWS - 1 of D (zero rows from `end` on) into a staged tile; wide: D is 16-byte aligned
template <int ROWS, int NTH>
__device__ __forceinline__ void bf_stage(unsigned char* tile, const uint8_t* __restrict__ D, int r0, int end, bool wide) {
#pragma unroll
    for (int e = threadIdx.x; e < ROWS * 8; e += NTH) {
        const int r = e >> 3, q = e & 7;
        unsigned char* dst = tile + r * BF_PITCH + q * 16;
        if (r0 + r < end)
            bf_cp_async(dst, D + (size_t)(r0 + r) * 128 + q * 16, wide);
        else
            *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// squared norms of the staged rows (threads 2r, 2r + 1 take a half each); rows from `live` on get a
// value above every distance
template <int ROWS, int NTH>
__device__ __forceinline__ void bf_norms(const unsigned char* tile, int live, int* out) {
    for (int e = threadIdx.x; e < ROWS * 2; e += NTH) {
        const uint4* p = reinterpret_cast<const uint4*>(tile + (e >> 1) * BF_PITCH + (e & 1) * 64);
        unsigned s = 0;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
            const uint4 w = p[v];
            s = __dp4a(w.x, w.x, s);
            s = __dp4a(w.y, w.y, s);
            s = __dp4a(w.z, w.z, s);
            s = __dp4a(w.w, w.w, s);
        }
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if ((e & 1) == 0) out[e >> 1] = (e >> 1) < live ? (int)s : 0x3fffffff;
    }
}

// One dense problem of a batch (an array in device memory, or one by value).
struct BfPair {
    const uint8_t *a, *b;
    Top2* part;                // splits x na
    unsigned long long* key;   // nb one-to-one keys
    int64_t *q, *t;
    int32_t* n;
    int na, nb, split_len, splits;
    int item0;                 // first CTA of the pair in the batch's grid
};

// the pair a CTA works on: the last one whose first item is not after `item`
__device__ __forceinline__ int bf_find(const BfPair* __restrict__ tab, int n, int item) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (tab[mid].item0 <= item) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// A CTA per (row block of 32 WR queries, split of B) of every pair: it sweeps B rows [n0, n1) for its
// queries and writes the per-row top-2 of its split. Squared distances of uint8 rows are integers below
// 2^24: four products and their sum per dp4a in 32-bit integers give exactly the values that float32
// multiply-adds give, a row's 128 bytes stay bytes in shared memory, and a thread's 8 x 8 block
// reads 16 bytes of 16 rows per 256 dp4a. The query norm is added once at the end (it is the same for
// every target of a row), and eight columns enter the running top-2 only when their smallest distance
// beats the second best, which happens a few times per row.
// Bound by the dp4a rate (half that of a multiply-add, four products each). Four pairs of about
// 7000 x 7000: 2318 -> 667 us for the whole call against float32 multiply-adds on tiles converted to
// float in shared memory, one pair after another; 1500 x 1500 from host arrays: 183 -> 102 us.
template <int WR>
__global__ void __launch_bounds__(64 * WR, WR == 4 ? 2 : 4)
    k_bf_exact(const __grid_constant__ BfPair one, const BfPair* __restrict__ tab, int n_pairs) {
    constexpr int BM = 32 * WR, NTH = 64 * WR;
    extern __shared__ __align__(16) unsigned char bf_sm[];
    unsigned char* sA = bf_sm;                                  // BM rows
    unsigned char* sB = bf_sm + BM * BF_PITCH;                  // two tiles of BN rows
    int* s_nb = reinterpret_cast<int*>(sB + 2 * BN * BF_PITCH);   // two tiles' norms
    int* s_na = s_nb + 2 * BN;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row0 = (warp >> 1) * 32 + (lane >> 3), col0 = (warp & 1) * 64 + (lane & 7);
    const BfPair& P = tab ? tab[bf_find(tab, n_pairs, blockIdx.x)] : one;
    const uint8_t* __restrict__ A = P.a;
    const uint8_t* __restrict__ B = P.b;
    const int na = P.na, item = blockIdx.x - P.item0, split = item % P.splits;
    const int m0 = (item / P.splits) * BM;
    const int n_begin = split * P.split_len;
    const int n_end = min(P.nb, n_begin + P.split_len);
    const bool wa = (reinterpret_cast<uintptr_t>(A) & 15) == 0, wb = (reinterpret_cast<uintptr_t>(B) & 15) == 0;
    bf_stage<BM, NTH>(sA, A, m0, na, wa);
    bf_stage<BN, NTH>(sB, B, n_begin, n_end, wb);
    int b1[8], b2[8], i1[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        b1[i] = b2[i] = 0x3fffffff;
        i1[i] = -1;
    }
    const unsigned char* pa = sA + row0 * BF_PITCH;
    int buf = 0;
    for (int n0 = n_begin; n0 < n_end; n0 += BN, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();   // this tile is in; every thread is done with the other one
        const unsigned char* tile = sB + buf * BN * BF_PITCH;
        if (n0 + BN < n_end) bf_stage<BN, NTH>(sB + (buf ^ 1) * BN * BF_PITCH, B, n0 + BN, n_end, wb);
        bf_norms<BN, NTH>(tile, n_end - n0, s_nb + buf * BN);
        const unsigned char* pb = tile + col0 * BF_PITCH;
        unsigned acc[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = 0u;
#pragma unroll 2
        for (int k = 0; k < 128; k += 8) {
            uint2 a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const uint2*>(pa + 4 * i * BF_PITCH + k);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint2 b = *reinterpret_cast<const uint2*>(pb + 8 * j * BF_PITCH + k);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = __dp4a(a[i].x, b.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[i][j] = __dp4a(a[i].y, b.y, acc[i][j]);
            }
        }
        __syncthreads();   // the tile's norms
        int cn[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) cn[j] = s_nb[buf * BN + col0 + 8 * j];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            int d[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) d[j] = cn[j] - 2 * (int)acc[i][j];
            const int m = min(min(min(d[0], d[1]), min(d[2], d[3])), min(min(d[4], d[5]), min(d[6], d[7])));
            if (m < b2[i]) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const bool less = d[j] < b1[i];
                    b2[i] = min(b2[i], max(b1[i], d[j]));
                    b1[i] = less ? d[j] : b1[i];
                    i1[i] = less ? n0 + col0 + 8 * j : i1[i];
                }
            }
        }
    }
    // merge the 16 column groups of each row through shared memory (the staged targets are dead)
    bf_norms<BM, NTH>(sA, BM, s_na);
    __syncthreads();
    int3 (*red)[BM] = reinterpret_cast<int3 (*)[BM]>(sB);
    static_assert(sizeof(int3) * 16 * BM <= 2 * BN * BF_PITCH, "merge area");
    const int grp = (warp & 1) * 8 + (lane & 7);
#pragma unroll
    for (int i = 0; i < 8; ++i) red[grp][row0 + 4 * i] = make_int3(b1[i], b2[i], i1[i]);
    __syncthreads();
    if (tid < BM && m0 + tid < na) {
        const float norm = (float)s_na[tid];
        Top2 t{INFINITY, INFINITY, -1};
        for (int g = 0; g < 16; ++g) {
            const int3 v = red[g][tid];
            Top2 o{INFINITY, INFINITY, v.z};
            if (v.x < 0x20000000) o.b1 = norm + (float)v.x;   // exact: integers below 2^24
            if (v.y < 0x20000000) o.b2 = norm + (float)v.y;
            t = top2_merge(t, o);
        }
        P.part[(size_t)split * na + m0 + tid] = t;
    }
}

template <int WR>
constexpr int bf_smem() {
    return 32 * WR * BF_PITCH + 2 * BN * BF_PITCH + (2 * BN + 32 * WR) * 4;
}

// How a batch of dense problems is cut into CTAs: WR = 4 (128 queries per CTA) once the 128 x 128 tiles
// outnumber two per SM, else WR = 2 (twice the CTAs); every pair's targets in splits of `tps` tiles,
// the number that gives the shortest schedule (waves of resident CTAs x (tiles + 1 for a CTA's
// own staging and merge)), bounded by the top-2 table's capacity.
struct BfPlan {
    int wr, tps, items;
    size_t parts;   // top-2 records
};
BfPlan bf_plan(const int* na, const int* nb, int n, size_t max_parts) {
    auto tiles = [&](int p) { return (nb[p] + BN - 1) / BN; };
    long long units = 0;
    int most = 1;
    for (int p = 0; p < n; ++p) {
        units += (long long)((na[p] + 127) / 128) * tiles(p);
        most = std::max(most, tiles(p));
    }
    BfPlan best{};
    best.wr = units >= 2 * 148 ? 4 : 2;
    const int bm = 32 * best.wr, slots = best.wr == 4 ? 2 * 148 : 4 * 148;
    double cost = 0.0;
    // with many tiles, finer steps than 1/64 of the longest sweep change little
    for (int tps = most; tps >= 1; tps -= std::max(1, tps / 64)) {
        long long items = 0;
        size_t parts = 0;
        for (int p = 0; p < n; ++p) {
            const long long sp = (tiles(p) + tps - 1) / tps;
            items += sp * ((na[p] + bm - 1) / bm);
            parts += (size_t)sp * na[p];
        }
        if (parts > max_parts || items > 0x7fffffffLL) break;   // more splits from here on
        const double c = (double)((items + slots - 1) / slots) * (tps + 1.0);
        if (best.tps == 0 || c < cost) {
            best.tps = tps;
            best.items = (int)items;
            best.parts = parts;
            cost = c;
        }
    }
    return best;
}
// fills p's split and first item; returns the next pair's first item
int bf_place(const BfPlan& pl, BfPair& p, int item0) {
    const int tiles = (p.nb + BN - 1) / BN, bm = 32 * pl.wr;
    p.split_len = pl.tps * BN;
    p.splits = (tiles + pl.tps - 1) / pl.tps;
    p.item0 = item0;
    return item0 + p.splits * ((p.na + bm - 1) / bm);
}

// The id of the current CUDA context, never given twice in a process (a context made after cudaDeviceReset
// gets the old one's handle); 0 if it cannot be queried. By the runtime's driver entry points, so that the
// library needs no link against libcuda.
unsigned long long context_id() {
    typedef int (*CtxGetCurrent)(void**);
    typedef int (*CtxGetId)(void*, unsigned long long*);
    auto entry = [](const char* name) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        return cudaGetDriverEntryPoint(name, &f, cudaEnableDefault, &q) == cudaSuccess &&
                       q == cudaDriverEntryPointSuccess ? f : nullptr;
    };
    static const CtxGetCurrent get = reinterpret_cast<CtxGetCurrent>(entry("cuCtxGetCurrent"));
    static const CtxGetId id_of = reinterpret_cast<CtxGetId>(entry("cuCtxGetId"));
    void* c = nullptr;
    unsigned long long id = 0;
    if (!get || !id_of || get(&c) != 0 || !c || id_of(c, &id) != 0) return 0;
    return id;
}

int32_t launch_bf(const BfPlan& pl, const BfPair& one, const BfPair* tab, int n, cudaStream_t s) {
    static_assert(bf_smem<2>() <= 48 * 1024, "needs no attribute");
    if (pl.wr == 4) {
        // the attribute belongs to the context: set again in one made after cudaDeviceReset
        static std::atomic<unsigned long long> set[64];
        int dev = 0;
        FSB_CUDA(cudaGetDevice(&dev));
        const unsigned long long id = context_id();
        if (id == 0 || dev >= 64 || set[dev].load(std::memory_order_acquire) != id) {
            FSB_CUDA(cudaFuncSetAttribute((const void*)k_bf_exact<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          bf_smem<4>()));
            if (dev < 64) set[dev].store(id, std::memory_order_release);
        }
        k_bf_exact<4><<<pl.items, 256, bf_smem<4>(), s>>>(one, tab, n);
    } else {
        k_bf_exact<2><<<pl.items, 128, bf_smem<2>(), s>>>(one, tab, n);
    }
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

// merge the splits, ratio test (float32, app/planesite/matching.py:96-99), one-to-one key of the target
__global__ void k_bf_merge(const __grid_constant__ BfPair one, const BfPair* __restrict__ tab, float ratio) {
    const BfPair& P = tab ? tab[blockIdx.y] : one;
    const int r = blockIdx.x * blockDim.x + threadIdx.x, na = P.na;
    if (r >= na) return;
    Top2 t = P.part[r];
    for (int s = 1; s < P.splits; ++s) t = top2_merge(t, P.part[(size_t)s * na + r]);
    const float b1 = fmaxf(t.b1, 0.f), b2 = fmaxf(t.b2, 0.f);
    const bool ok = __fsqrt_rn(b1) < __fmul_rn(ratio, __fsqrt_rn(b2));
    if (ok && t.i1 >= 0) atomicMin(P.key + t.i1, ((unsigned long long)(uint32_t)b1 << 32) | (unsigned)r);
}

// ------------------------------------------------------------------------------ one-to-one
__global__ void k_unique_keys(const int32_t* __restrict__ t_row, const uint32_t* __restrict__ d_row, int na,
                              unsigned long long* __restrict__ key) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= na) return;
    const int t = t_row[r];
    if (t >= 0) atomicMin(key + t, ((unsigned long long)d_row[r] << 32) | (unsigned)r);
}

__global__ void __launch_bounds__(COMPACT_T) k_unique_compact(const unsigned long long* __restrict__ key, int nb,
                                                              int64_t* __restrict__ q, int64_t* __restrict__ t,
                                                              int32_t* __restrict__ n_out) {
    unique_compact(key, nb, q, t, n_out);
}
// a block per pair of a batch
__global__ void __launch_bounds__(COMPACT_T) k_bf_compact(const BfPair* __restrict__ tab) {
    const BfPair& P = tab[blockIdx.x];
    unique_compact(P.key, P.nb, P.q, P.t, P.n);
}

__global__ void k_unique_flags(const unsigned long long* __restrict__ key, int nb, uint8_t* __restrict__ flag,
                               int32_t* __restrict__ iota) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb) return;
    flag[t] = key[t] != ~0ull;
    iota[t] = t;
}

__global__ void k_unique_emit(const unsigned long long* __restrict__ key, const int32_t* __restrict__ tsel,
                              const int* __restrict__ n, int64_t* __restrict__ q, int64_t* __restrict__ t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *n) return;
    const int tt = tsel[i];
    q[i] = (int64_t)(key[tt] & 0xffffffffull);
    t[i] = tt;
}

// ------------------------------------------------------------------------------ guided
struct GridSpec {
    double x0, y0, cs;   // origin and cell size
    int gw, gh;
};

__device__ __forceinline__ int cell_of(double v, double o, double cs, int n) {
    const double f = floor((v - o) / cs);
    return f < 0.0 ? 0 : (f >= (double)(n - 1) ? n - 1 : (int)f);
}

constexpr int G_WARPS = 4, G_CAND = 512;

// One pair of a guided batch (an array in device memory, or one by value).
struct GPair {
    const double* pred;
    const uint8_t* a;
    const double* bxy;
    const uint8_t* b;
    int na, nb;
    double wb, hb;
    GridSpec gs;
    int cell0;   // first cell of this pair's grid
    int item0;   // first target (B row) in the concatenated target arrays
    int64_t* q_out;
    int64_t* t_out;
    int32_t* n_out;
};

__global__ void k_gb_count(const __grid_constant__ GPair one, const GPair* __restrict__ tab, int32_t* __restrict__ cell,
                           int32_t* __restrict__ count) {
    const GPair& P = tab ? tab[blockIdx.y] : one;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= P.nb) return;
    const int cx = cell_of(P.bxy[2 * j], P.gs.x0, P.gs.cs, P.gs.gw), cy = cell_of(P.bxy[2 * j + 1], P.gs.y0, P.gs.cs, P.gs.gh);
    const int c = P.cell0 + cy * P.gs.gw + cx;
    cell[P.item0 + j] = c;
    atomicAdd(count + c, 1);
}

// targets in cell order: index and position
__global__ void k_gb_fill(const __grid_constant__ GPair one, const GPair* __restrict__ tab, const int32_t* __restrict__ cell,
                          const int32_t* __restrict__ start, int32_t* __restrict__ cursor, int32_t* __restrict__ items,
                          double2* __restrict__ pos) {
    const GPair& P = tab ? tab[blockIdx.y] : one;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= P.nb) return;
    const int c = cell[P.item0 + j];
    const int at = start[c] + atomicAdd(cursor + c, 1);
    items[at] = j;   // local target index
    pos[at] = make_double2(P.bxy[2 * j], P.bxy[2 * j + 1]);
}

__device__ __forceinline__ void top2_push_tie(Top2& t, float d, int j) {   // equal distances: smaller index
    if (d < t.b1 || (d == t.b1 && j < t.i1)) {
        t.b2 = t.b1;
        t.b1 = d;
        t.i1 = j;
    } else if (d < t.b2) {
        t.b2 = d;
    }
}

// exact squared distances of the query row (16-byte segment a4 of this lane, squared norm qn) to the m
// targets of `list`, into this lane's top-2: eight lanes per target, one 16-byte load each, and
// |b|^2 - 2 a.b summed over the eight; eight targets in flight
__device__ __forceinline__ void guided_distances(const uint4& a4, int qn, const uint8_t* __restrict__ B,
                                                 const int32_t* list, int m, Top2& best) {
    const int lane = threadIdx.x & 31, seg = lane & 7, g = lane >> 3;
    for (int c0 = 0; c0 < m; c0 += 8) {
        int j[2], v[2];
        uint4 b[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            j[u] = list[min(c0 + 4 * u + g, m - 1)];
            b[u] = __ldg(reinterpret_cast<const uint4*>(B + (size_t)j[u] * 128) + seg);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            unsigned ab = __dp4a(a4.x, b[u].x, 0u), bb = __dp4a(b[u].x, b[u].x, 0u);
            ab = __dp4a(a4.y, b[u].y, ab);
            bb = __dp4a(b[u].y, b[u].y, bb);
            ab = __dp4a(a4.z, b[u].z, ab);
            bb = __dp4a(b[u].z, b[u].z, bb);
            ab = __dp4a(a4.w, b[u].w, ab);
            bb = __dp4a(b[u].w, b[u].w, bb);
            v[u] = (int)bb - 2 * (int)ab;
#pragma unroll
            for (int sh = 1; sh < 8; sh <<= 1) v[u] += __shfl_xor_sync(0xffffffffu, v[u], sh);
            if (c0 + 4 * u + g < m) top2_push_tie(best, (float)(qn + v[u]), j[u]);
        }
    }
}

// Guided matcher, one warp per query: the candidates of the prior window, exact distances, top-2, ratio
// test and the one-to-one key of the target; or (c_t set) the best candidate before the ratio test.
// The three grid rows of the window are three contiguous runs of the cell-ordered targets, so the
// window is one list read 32 positions at a time (about 25 at 9000 targets of a 2640 x 1978 frame and
// a radius of 40) instead of nine cells one after another, and a candidate's row is one coalesced
// 128-byte read instead of eight strided ones.
// Bound by the latency of the dependent reads (cell starts, positions, rows). 64 pairs of 2000-16000
// features: 1219 us with nine cells and a lane per candidate (plus 188 us for norms), 404 us now.
__global__ void __launch_bounds__(G_WARPS * 32) k_gb_guided(const __grid_constant__ GPair one, const GPair* __restrict__ tab,
                                                            const int32_t* __restrict__ start,
                                                            const int32_t* __restrict__ items,
                                                            const double2* __restrict__ pos, double radius, int kc,
                                                            float ratio, int per_block,
                                                            unsigned long long* __restrict__ key,
                                                            int32_t* __restrict__ c_t, float* __restrict__ c_b12,
                                                            int* __restrict__ overflow) {
    __shared__ double s_cd[G_WARPS][G_CAND];
    __shared__ int32_t s_ci[G_WARPS][G_CAND];
    const GPair& P = tab ? tab[blockIdx.y] : one;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31, seg = lane & 7;
    double* cd = s_cd[wid];
    int32_t* ci = s_ci[wid];
    const unsigned lt = (1u << lane) - 1u;
    const bool wide = (reinterpret_cast<uintptr_t>(P.a) & 15) == 0;
    const int q1 = min(P.na, (int)(blockIdx.x + 1) * per_block);
    for (int q = blockIdx.x * per_block + wid; q < q1; q += G_WARPS) {
        const double px = P.pred[2 * (size_t)q], py = P.pred[2 * (size_t)q + 1];
        Top2 best{INFINITY, INFINITY, -1};
        if (px > -radius && px < P.wb + radius && py > -radius && py < P.hb + radius) {
            uint4 a4;
            const uint8_t* ar = P.a + (size_t)q * 128 + seg * 16;
            if (wide) {
                a4 = __ldg(reinterpret_cast<const uint4*>(ar));
            } else {
                const uint32_t* aw = reinterpret_cast<const uint32_t*>(ar);
                a4 = make_uint4(__ldg(aw), __ldg(aw + 1), __ldg(aw + 2), __ldg(aw + 3));
            }
            const int cx = cell_of(px, P.gs.x0, P.gs.cs, P.gs.gw), cy = cell_of(py, P.gs.y0, P.gs.cs, P.gs.gh);
            // lane r < 3: the run of grid row cy - 1 + r
            int s0 = 0, len = 0;
            const int yy = cy - 1 + lane;
            if (lane < 3 && yy >= 0 && yy < P.gs.gh) {
                const int32_t* row = start + P.cell0 + yy * P.gs.gw;
                s0 = row[max(cx - 1, 0)];
                len = row[min(cx + 1, P.gs.gw - 1) + 1] - s0;
            }
            const int l0 = __shfl_sync(0xffffffffu, len, 0), l1 = __shfl_sync(0xffffffffu, len, 1);
            const int l2 = __shfl_sync(0xffffffffu, len, 2);
            // slot of the window's e-th target: e + the offset of its run
            const int o0 = __shfl_sync(0xffffffffu, s0, 0), o1 = __shfl_sync(0xffffffffu, s0, 1) - l0;
            const int o2 = __shfl_sync(0xffffffffu, s0, 2) - l0 - l1;
            const int n = l0 + l1 + l2;
            unsigned qn = __dp4a(a4.x, a4.x, 0u);
            qn = __dp4a(a4.y, a4.y, qn);
            qn = __dp4a(a4.z, a4.z, qn);
            qn = __dp4a(a4.w, a4.w, qn);
#pragma unroll
            for (int sh = 1; sh < 8; sh <<= 1) qn += __shfl_xor_sync(0xffffffffu, qn, sh);
            const double r2 = radius * radius;
            int cnt = 0;
            for (int e0 = 0; e0 < n; e0 += 32) {
                const int e = e0 + lane;
                bool hit = false;
                double d2 = 0.0;
                int j = 0;
                if (e < n) {
                    const int at = e + (e < l0 ? o0 : e < l0 + l1 ? o1 : o2);
                    j = __ldg(items + at);
                    const double2 p = __ldg(pos + at);
                    const double dx = __dsub_rn(p.x, px), dy = __dsub_rn(p.y, py);
                    d2 = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
                    hit = d2 < r2;
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const int at = cnt + __popc(m & lt);
                    if (at < G_CAND) {
                        cd[at] = d2;
                        ci[at] = j;
                    }
                }
                cnt += __popc(m);
                if (kc <= 0) {   // every target strictly within the radius: no list to keep
                    __syncwarp();
                    guided_distances(a4, (int)qn, P.b, ci, cnt, best);
                    __syncwarp();
                    cnt = 0;
                }
            }
            __syncwarp();
            if (kc > 0) {
                if (cnt > G_CAND) {
                    if (lane == 0) atomicExch(overflow, 1);
                    cnt = G_CAND;
                }
                if (cnt > kc) {
                    // keep the kc nearest (ties: smaller B index): bit c of `keep` is entry 32 c + lane
                    unsigned keep = 0;
                    for (int e = lane, c = 0; e < cnt; e += 32, ++c) {
                        const double de = cd[e];
                        const int ie = ci[e];
                        int rank = 0;
                        for (int f = 0; f < cnt; ++f) {
                            const double df = cd[f];
                            rank += (df < de || (df == de && ci[f] < ie)) ? 1 : 0;
                        }
                        if (rank < kc) keep |= 1u << c;
                    }
                    __syncwarp();
                    int kept = 0;
                    for (int e0 = 0, c = 0; e0 < cnt; e0 += 32, ++c) {
                        const bool k = keep >> c & 1u;
                        const int j = k ? ci[e0 + lane] : 0;
                        const unsigned m = __ballot_sync(0xffffffffu, k);
                        if (k) ci[kept + __popc(m & lt)] = j;   // at or before its own entry
                        kept += __popc(m);
                        __syncwarp();
                    }
                    cnt = kept;
                }
                if (cnt > 0) guided_distances(a4, (int)qn, P.b, ci, cnt, best);
                __syncwarp();
            }
            // merge the four groups' top-2
#pragma unroll
            for (int sh = 8; sh < 32; sh <<= 1) {
                Top2 o;
                o.b1 = __shfl_xor_sync(0xffffffffu, best.b1, sh);
                o.b2 = __shfl_xor_sync(0xffffffffu, best.b2, sh);
                o.i1 = __shfl_xor_sync(0xffffffffu, best.i1, sh);
                best = top2_merge(best, o);
            }
        }
        if (lane == 0) {
            if (c_t) {   // the best candidate before the ratio test (learned filter input)
                c_t[q] = best.i1;
                c_b12[2 * (size_t)q] = best.b1;
                c_b12[2 * (size_t)q + 1] = best.b2;
            } else if (best.i1 >= 0 && __fsqrt_rn(best.b1) < __fmul_rn(ratio, __fsqrt_rn(best.b2))) {
                // single candidate: b2 = inf passes (app/planesite/matching.py:142-146)
                atomicMin(key + P.item0 + best.i1, ((unsigned long long)(uint32_t)best.b1 << 32) | (unsigned)q);
            }
        }
    }
}

// matches of each pair ordered by target: a block per pair
__global__ void __launch_bounds__(COMPACT_T) k_gb_compact(const __grid_constant__ GPair one, const GPair* __restrict__ tab,
                                                          const unsigned long long* __restrict__ key) {
    const GPair& P = tab ? tab[blockIdx.x] : one;
    unique_compact(key + P.item0, P.nb, P.q_out, P.t_out, P.n_out);
}

__global__ void k_perspective(const double* __restrict__ xy, int n, const double* __restrict__ hm,
                              double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = xy[2 * i], y = xy[2 * i + 1];
    double w = __dadd_rn(__dadd_rn(__dmul_rn(hm[6], x), __dmul_rn(hm[7], y)), hm[8]);
    double u = 0.0, v = 0.0;
    if (fabs(w) > 1.1920928955078125e-07) {
        w = 1.0 / w;
        u = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(hm[0], x), __dmul_rn(hm[1], y)), hm[2]), w);
        v = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(hm[3], x), __dmul_rn(hm[4], y)), hm[5]), w);
    }
    out[2 * i] = u;
    out[2 * i + 1] = v;
}

// the one-to-one keys of nb targets -> matches ordered by target: q[i], t[i], *d_n
int32_t emit_unique(fsb_ctx* ctx, const unsigned long long* key, int nb, int64_t* d_q, int64_t* d_t, int* d_n,
                    cudaStream_t s) {
    if (nb <= kCompactMax) {
        k_unique_compact<<<1, COMPACT_T, 0, s>>>(key, nb, d_q, d_t, d_n);
        note_launch();
        FSB_CUDA(cudaGetLastError());
        return FSB_OK;
    }
    FSB_TRY(ctx->s_misc2.ensure((size_t)nb * 9 + 1024));
    uint8_t* flag = ctx->s_misc2.as<uint8_t>();
    int32_t* iota = reinterpret_cast<int32_t*>(flag + ((nb + 255) / 256) * 256);
    int32_t* tsel = iota + nb;
    k_unique_flags<<<blocks(nb, 256), 256, 0, s>>>(key, nb, flag, iota);
    size_t tb = 0;
    cub::DeviceSelect::Flagged(nullptr, tb, iota, flag, tsel, d_n, nb, s);
    FSB_TRY(ctx->s_cub.ensure(tb + 16));
    FSB_CUDA(cub::DeviceSelect::Flagged(ctx->s_cub.p, tb, iota, flag, tsel, d_n, nb, s));
    k_unique_emit<<<blocks(nb, 256), 256, 0, s>>>(key, tsel, d_n, d_q, d_t);
    note_launch(2);
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

// one-to-one filter + compaction ordered by target
int32_t run_unique(fsb_ctx* ctx, const int32_t* t_row, const uint32_t* d_row, int na, int nb, int64_t* d_q,
                   int64_t* d_t, int* d_n, cudaStream_t s) {
    FSB_TRY(ctx->s_u64.ensure((size_t)nb * 8 + 64));
    unsigned long long* key = ctx->s_u64.as<unsigned long long>();
    FSB_CUDA(cudaMemsetAsync(key, 0xff, (size_t)nb * 8, s));
    k_unique_keys<<<blocks(na, 256), 256, 0, s>>>(t_row, d_row, na, key);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return emit_unique(ctx, key, nb, d_q, d_t, d_n, s);
}

__device__ __forceinline__ uint32_t orderable(float f) {
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__global__ void k_uq_keys1(const float* __restrict__ dd, int n, uint32_t* __restrict__ key, uint32_t* __restrict__ val) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = orderable(dd[i]);
    val[i] = (uint32_t)i;
}

__global__ void k_uq_keys2(const int64_t* __restrict__ t, const uint32_t* __restrict__ perm, int n,
                           unsigned long long* __restrict__ key) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = (unsigned long long)t[perm[i]] ^ 0x8000000000000000ull;
}

__global__ void k_uq_first(const unsigned long long* __restrict__ key, int n, uint8_t* __restrict__ flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flag[i] = (i == 0 || key[i] != key[i - 1]) ? 1 : 0;
}

__global__ void k_uq_emit(const uint32_t* __restrict__ pos, const int* __restrict__ n, const int64_t* __restrict__ q,
                          const int64_t* __restrict__ t, int64_t* __restrict__ qo, int64_t* __restrict__ to) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *n) return;
    qo[i] = q[pos[i]];
    to[i] = t[pos[i]];
}


}  // namespace

// General one-to-one filter (matching._unique) for arbitrary int64 targets and float distances:
// stable sorts by distance then by target give (t, dd, position) order; the first of each target
// run is kept.
int32_t run_unique_general(fsb_ctx* ctx, const int64_t* d_q, const int64_t* d_t, const float* d_dd, int n,
                           int64_t* d_qo, int64_t* d_to, int* d_n, cudaStream_t s) {
    const size_t N = (size_t)n;
    FSB_TRY(ctx->s_misc.ensure(N * (4 * 4 + 8 * 2 + 1 + 4) + 256));
    uint32_t* k1 = ctx->s_misc.as<uint32_t>();
    uint32_t* k1o = k1 + N;
    uint32_t* v1 = k1o + N;
    uint32_t* v1o = v1 + N;
    unsigned long long* k2 = reinterpret_cast<unsigned long long*>(v1o + N);
    unsigned long long* k2o = k2 + N;
    uint32_t* v2o = reinterpret_cast<uint32_t*>(k2o + N);
    uint8_t* flag = reinterpret_cast<uint8_t*>(v2o + N);
    uint32_t* sel = v1;   // reused after the second sort
    size_t t1 = 0, t2 = 0, t3 = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, t1, k1, k1o, v1, v1o, n, 0, 32, s);
    cub::DeviceRadixSort::SortPairs(nullptr, t2, k2, k2o, v1o, v2o, n, 0, 64, s);
    cub::DeviceSelect::Flagged(nullptr, t3, v2o, flag, sel, d_n, n, s);
    size_t tmax = t1 > t2 ? t1 : t2;
    tmax = tmax > t3 ? tmax : t3;
    FSB_TRY(ctx->s_cub.ensure(tmax + 16));
    k_uq_keys1<<<blocks(n, 256), 256, 0, s>>>(d_dd, n, k1, v1);
    size_t tb = tmax;
    FSB_CUDA(cub::DeviceRadixSort::SortPairs(ctx->s_cub.p, tb, k1, k1o, v1, v1o, n, 0, 32, s));
    k_uq_keys2<<<blocks(n, 256), 256, 0, s>>>(d_t, v1o, n, k2);
    tb = tmax;
    FSB_CUDA(cub::DeviceRadixSort::SortPairs(ctx->s_cub.p, tb, k2, k2o, v1o, v2o, n, 0, 64, s));
    k_uq_first<<<blocks(n, 256), 256, 0, s>>>(k2o, n, flag);
    tb = tmax;
    FSB_CUDA(cub::DeviceSelect::Flagged(ctx->s_cub.p, tb, v2o, flag, sel, d_n, n, s));
    k_uq_emit<<<blocks(n, 256), 256, 0, s>>>(sel, d_n, d_q, d_t, d_qo, d_to);
    note_launch(4);
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

struct H9 {
    double h[9];
};

// float32 points -> float64 positions through a homography, plus optional float32 offsets
__global__ void k_project(const float* __restrict__ xy, int n, H9 H, const float* __restrict__ off,
                          double* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double x = (double)xy[2 * i], y = (double)xy[2 * i + 1];
    const double* hm = H.h;
    double w = __dadd_rn(__dadd_rn(__dmul_rn(hm[6], x), __dmul_rn(hm[7], y)), hm[8]);
    double u = 0.0, v = 0.0;
    if (fabs(w) > 1.1920928955078125e-07) {
        w = 1.0 / w;
        u = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(hm[0], x), __dmul_rn(hm[1], y)), hm[2]), w);
        v = __dmul_rn(__dadd_rn(__dadd_rn(__dmul_rn(hm[3], x), __dmul_rn(hm[4], y)), hm[5]), w);
    }
    if (off) {
        u += (double)off[2 * i];
        v += (double)off[2 * i + 1];
    }
    out[2 * i] = u;
    out[2 * i + 1] = v;
}

int32_t run_project(const float* d_xy, int n, const double* hm9, const float* d_off, double* d_out, cudaStream_t s) {
    if (n <= 0) return FSB_OK;
    H9 H;
    for (int i = 0; i < 9; ++i) H.h[i] = hm9[i];
    k_project<<<blocks(n, 256), 256, 0, s>>>(d_xy, n, H, d_off, d_out);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

int32_t run_perspective(const double* d_xy, int n, const double* d_hm9, double* d_out, cudaStream_t s) {
    if (n <= 0) return FSB_OK;
    k_perspective<<<blocks(n, 256), 256, 0, s>>>(d_xy, n, d_hm9, d_out);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

int32_t run_match_bf(fsb_ctx* ctx, const uint8_t* d_a, int na, const uint8_t* d_b, int nb, float ratio,
                     int precision, int64_t* d_q, int64_t* d_t, int* d_n, cudaStream_t s) {
    if (na < 2 || nb < 2) {
        FSB_CUDA(cudaMemsetAsync(d_n, 0, sizeof(int), s));
        return FSB_OK;
    }
    if (precision != FSB_PREC_FP32)
        return run_match_bf_tc(ctx, 1, &d_a, &na, &d_b, &nb, ratio, precision, &d_q, &d_t, d_n, nullptr,
                               &ctx->tc_stats, s);
    const BfPlan pl = bf_plan(&na, &nb, 1, (size_t)1 << 40);
    FSB_TRY(ctx->s_misc.ensure(pl.parts * sizeof(Top2) + 64));
    FSB_TRY(ctx->s_u64.ensure((size_t)nb * 8 + 64));
    BfPair one{d_a, d_b, ctx->s_misc.as<Top2>(), ctx->s_u64.as<unsigned long long>(), d_q, d_t, d_n, na, nb};
    bf_place(pl, one, 0);
    FSB_CUDA(cudaMemsetAsync(one.key, 0xff, (size_t)nb * 8, s));
    FSB_TRY(launch_bf(pl, one, nullptr, 1, s));
    k_bf_merge<<<blocks(na, 256), 256, 0, s>>>(one, nullptr, ratio);
    note_launch();
    FSB_CUDA(cudaGetLastError());
    return emit_unique(ctx, one.key, nb, d_q, d_t, d_n, s);
}

// A batch of FP32 dense problems (each na, nb >= 2) in one set of launches: counts (device, one per
// pair). Pairs with more targets than one block compacts run one after another instead.
int32_t run_match_bf_batch(fsb_ctx* ctx, int n, const uint8_t* const* d_a, const int* na, const uint8_t* const* d_b,
                           const int* nb, float ratio, int64_t* const* d_q, int64_t* const* d_t, int32_t* counts,
                           cudaStream_t s) {
    bool one_by_one = n == 1 || n > 65535;   // a grid's second dimension
    for (int p = 0; p < n; ++p) one_by_one = one_by_one || nb[p] > kCompactMax;
    if (one_by_one) {
        for (int p = 0; p < n; ++p)
            FSB_TRY(run_match_bf(ctx, d_a[p], na[p], d_b[p], nb[p], ratio, FSB_PREC_FP32, d_q[p], d_t[p], counts + p, s));
        return FSB_OK;
    }
    const BfPlan pl = bf_plan(na, nb, n, (size_t)1 << 40);
    size_t keys = 0;
    int max_na = 0;
    for (int p = 0; p < n; ++p) {
        keys += (size_t)nb[p];
        max_na = std::max(max_na, na[p]);
    }
    FSB_TRY(ctx->s_misc.ensure(pl.parts * sizeof(Top2) + 64));
    FSB_TRY(ctx->s_u64.ensure(keys * 8 + 64));
    FSB_TRY(ctx->s_i32.ensure((size_t)n * sizeof(BfPair)));
    std::vector<BfPair> tab(n);
    Top2* part = ctx->s_misc.as<Top2>();
    unsigned long long* key = ctx->s_u64.as<unsigned long long>();
    int item = 0;
    for (int p = 0; p < n; ++p) {
        tab[p] = BfPair{d_a[p], d_b[p], part, key, d_q[p], d_t[p], counts + p, na[p], nb[p]};
        item = bf_place(pl, tab[p], item);
        part += (size_t)tab[p].splits * na[p];
        key += nb[p];
    }
    BfPair* d_tab = ctx->s_i32.as<BfPair>();
    FSB_CUDA(cudaMemcpyAsync(d_tab, tab.data(), (size_t)n * sizeof(BfPair), cudaMemcpyHostToDevice, s));
    FSB_CUDA(cudaMemsetAsync(ctx->s_u64.p, 0xff, keys * 8, s));
    FSB_TRY(launch_bf(pl, tab[0], d_tab, n, s));
    k_bf_merge<<<dim3(blocks(max_na, 256), (unsigned)n), 256, 0, s>>>(tab[0], d_tab, ratio);
    k_bf_compact<<<n, COMPACT_T, 0, s>>>(d_tab);
    note_launch(2);
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}

int32_t run_unique_rows(fsb_ctx* ctx, const int32_t* t_row, const uint32_t* d_row, int na, int nb, int64_t* d_q,
                        int64_t* d_t, int* d_n, cudaStream_t s) {
    return run_unique(ctx, t_row, d_row, na, nb, d_q, d_t, d_n, s);
}

// Guided matching of a batch of pairs (each na, nb >= 1, radius > 0) with _unique in one set of
// launches: h_counts (host) receives the match count of each pair; the call waits. With c_t / c_b12
// (one pair only) the candidates before the ratio test are written instead. d_n: device, one per pair.
int32_t run_match_guided_batch(fsb_ctx* ctx, int n_pairs, const double* const* d_pred, const uint8_t* const* d_a,
                               const int* na, const double* const* d_bxy, const uint8_t* const* d_b, const int* nb,
                               const double* wb, const double* hb, double radius, int kc, float ratio,
                               int64_t* const* d_q, int64_t* const* d_t, int32_t* d_n, int32_t* h_counts, cudaStream_t s,
                               int32_t* c_t, float* c_b12) {
    if (n_pairs <= 0) return FSB_OK;
    std::vector<GPair> hp(n_pairs);
    long long cells = 0, rows = 0, items = 0;
    int max_na = 0, max_nb = 0;
    for (int p = 0; p < n_pairs; ++p) {
        GPair& P = hp[p];
        P.pred = d_pred[p];
        P.a = d_a[p];
        P.bxy = d_bxy[p];
        P.b = d_b[p];
        P.na = na[p];
        P.nb = nb[p];
        P.wb = wb[p];
        P.hb = hb[p];
        GridSpec gs;
        gs.x0 = 0.0;
        gs.y0 = 0.0;
        gs.cs = radius;
        double gwd = (wb[p] > 0 ? wb[p] : 1.0) / radius + 1.0, ghd = (hb[p] > 0 ? hb[p] : 1.0) / radius + 1.0;
        while (gwd * ghd > 4.0e6) {
            gs.cs *= 2.0;
            gwd = (wb[p] > 0 ? wb[p] : 1.0) / gs.cs + 1.0;
            ghd = (hb[p] > 0 ? hb[p] : 1.0) / gs.cs + 1.0;
        }
        gs.gw = (int)gwd;
        gs.gh = (int)ghd;
        P.gs = gs;
        P.cell0 = (int)cells;
        P.item0 = (int)items;
        P.q_out = d_q ? d_q[p] : nullptr;
        P.t_out = d_t ? d_t[p] : nullptr;
        P.n_out = d_n ? d_n + p : nullptr;
        cells += (long long)gs.gw * gs.gh;
        rows += na[p];
        items += nb[p];
        max_na = std::max(max_na, na[p]);
        max_nb = std::max(max_nb, nb[p]);
    }
    if (cells + items + rows > 0x7fffffffLL) {
        set_error("guided batch too large (%lld cells, %lld targets, %lld queries)", cells, items, rows);
        return FSB_ERR_ARG;
    }
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (int32_t*)nullptr, (int32_t*)nullptr, (int)(cells + 1), s);
    auto al = [](size_t x) { return (x + 255) & ~size_t(255); };
    const size_t b_pairs = n_pairs > 1 ? al((size_t)n_pairs * sizeof(GPair)) : 0, b_items = al((size_t)items * 4);
    const size_t b_cells = al((size_t)(cells + 1) * 4);
    FSB_TRY(ctx->s_gb.ensure(b_pairs + 2 * b_items + al((size_t)items * 16) + 3 * b_cells + 256 + al((size_t)items * 8) +
                             al(tb)));
    uint8_t* cur = ctx->s_gb.as<uint8_t>();
    auto take = [&](size_t bytes) {
        uint8_t* p = cur;
        cur += bytes;
        return p;
    };
    GPair* tab = n_pairs > 1 ? reinterpret_cast<GPair*>(take(b_pairs)) : nullptr;
    int32_t* cell = reinterpret_cast<int32_t*>(take(b_items));
    int32_t* gitems = reinterpret_cast<int32_t*>(take(b_items));
    double2* pos = reinterpret_cast<double2*>(take(al((size_t)items * 16)));
    int32_t* start = reinterpret_cast<int32_t*>(take(b_cells));
    int32_t* count = reinterpret_cast<int32_t*>(take(b_cells));    // count, cursor and the overflow
    int32_t* cursor = reinterpret_cast<int32_t*>(take(b_cells));   // flag are cleared together
    int* overflow = reinterpret_cast<int*>(take(256));
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(take(al((size_t)items * 8)));
    void* tmp = take(al(tb));
    if (tab) FSB_CUDA(cudaMemcpyAsync(tab, hp.data(), (size_t)n_pairs * sizeof(GPair), cudaMemcpyHostToDevice, s));
    FSB_CUDA(cudaMemsetAsync(count, 0, 2 * b_cells + 256, s));
    const unsigned py = (unsigned)n_pairs;
    k_gb_count<<<dim3(blocks(max_nb, 256), py), 256, 0, s>>>(hp[0], tab, cell, count);
    FSB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, tb, count, start, (int)(cells + 1), s));
    k_gb_fill<<<dim3(blocks(max_nb, 256), py), 256, 0, s>>>(hp[0], tab, cell, start, cursor, gitems, pos);
    if (!c_t) FSB_CUDA(cudaMemsetAsync(keys, 0xff, (size_t)items * 8, s));
    // Queries of a block of four warps. One per warp: the chains of dependent reads of up to 5 300 queries run at
    // once (one pair of 2000 x 2000, a radius of 400: 179 us with four per warp, one after another, 117 with one;
    // 9000 x 9000: 480 and 307). Photos' pairs of 7000, a radius of 100: 28 000 queries 206 and 192 us, 56 000 295 and
    // 287, 112 000 454 and 464; a radius of 40: 208 each at 56 000, 377 and 397 at 192 000. Full either way, the GPU
    // is faster with fewer and longer blocks.
    const int per_block = rows <= 64000 ? G_WARPS : 4 * G_WARPS;
    k_gb_guided<<<dim3(blocks(max_na, per_block), py), G_WARPS * 32, 0, s>>>(
        hp[0], tab, start, gitems, pos, radius, kc, ratio, per_block, keys, c_t, c_b12, overflow);
    note_launch(4);
    FSB_CUDA(cudaGetLastError());
    if (!c_t) {
        if (max_nb <= kCompactMax) {
            k_gb_compact<<<py, COMPACT_T, 0, s>>>(hp[0], tab, keys);
            note_launch();
            FSB_CUDA(cudaGetLastError());
        } else {
            for (const GPair& P : hp)
                FSB_TRY(emit_unique(ctx, keys + P.item0, P.nb, P.q_out, P.t_out, P.n_out, s));
        }
        if (h_counts) FSB_CUDA(cudaMemcpyAsync(h_counts, d_n, (size_t)n_pairs * 4, cudaMemcpyDeviceToHost, s));
    }
    int h_over = 0;
    FSB_CUDA(cudaMemcpyAsync(&h_over, overflow, sizeof(int), cudaMemcpyDeviceToHost, s));
    FSB_CUDA(cudaStreamSynchronize(s));
    if (h_over) {
        set_error("more than %d B keypoints within the radius of one prediction (kc mode)", G_CAND);
        return FSB_ERR_OVERFLOW;
    }
    return FSB_OK;
}

}  // namespace fsb

// ---------------------------------------------------------------------------------------------
// Allocation-free dense ratio matcher (fsb_match_bf_noalloc).
//
// Some callers cannot call cudaMalloc: services that reserve their whole device-memory budget
// when they start (a fixed pool handed to them by a host application, as in multi-tenant
// serving), host frameworks that own the CUDA allocator and forbid allocations behind their back,
// and real-time loops where an allocation may block or fail in the middle of a frame. For them
// this entry point runs the FP32 dense matcher with all of its scratch in one file-scope device
// array of fixed size (kNoAllocScratchBytes, about 1.6 MiB), so a call allocates nothing: the
// caller passes device inputs and outputs and a stream.
//
// The array lives in every GPU that loads this library until the process exits. Host code may
// not use its name as an address (on the host it is only a stand-in symbol), so its device
// address is looked up with cudaGetSymbolAddress, with that device current, by the first call made
// on the device (and again by the first call in another context of that device, e.g. after a
// cudaDeviceReset); that first call should come before any stream capture.
// Every call shares the array and it keeps the last call's contents: the per-target key table is
// re-filled at the start of each call, everything else is fully overwritten. Calls whose work
// overlaps on the GPU (different streams, or host threads using the same device) race on the
// array and must be serialised by the caller.
namespace fsb {
namespace {

constexpr int kNoAllocMaxRows = 16384;
constexpr int kNoAllocSplitRows = 8 * kNoAllocMaxRows;   // capacity of the per-split top-2 table
constexpr size_t kNoAllocScratchBytes =
    sizeof(unsigned long long) * kNoAllocMaxRows +         // one-to-one keys per target
    sizeof(Top2) * (size_t)kNoAllocSplitRows;              // per-split top-2 of every A row

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

std::mutex g_noalloc_mu;
void* g_noalloc_addr[256] = {};
unsigned long long g_noalloc_ctx[256] = {};   // the id of the CUDA context the cached address belongs to

// Device address of g_noalloc_scratch in the current device's current context. It is looked up
// on the first call in a context and cached with that context's id; a different context on
// the same device (the module loaded again after cudaDeviceReset, or a driver-API context other
// than the primary one) looks it up again.
int32_t noalloc_scratch(void** out) {
    int dev = 0;
    FSB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) {
        set_error("device ordinal %d out of range", dev);
        return FSB_ERR_ARG;
    }
    const unsigned long long ctx = context_id();
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev] || ctx == 0 || ctx != g_noalloc_ctx[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || p == nullptr) {
            set_error("cudaGetSymbolAddress(scratch) failed on device %d: %s", dev, cudaGetErrorString(e));
            return FSB_ERR_CUDA;
        }
        g_noalloc_addr[dev] = p;
        g_noalloc_ctx[dev] = ctx;
    }
    *out = g_noalloc_addr[dev];
    return FSB_OK;
}

}  // namespace
}  // namespace fsb

extern "C" int32_t fsb_match_bf_noalloc(const uint8_t* d_a, int32_t na, const uint8_t* d_b, int32_t nb,
                                        float ratio, int64_t* d_q, int64_t* d_t, int32_t* d_n, void* stream) {
    using namespace fsb;
    FSB_ARG(d_n != nullptr, "n_out is null");
    FSB_ARG(na >= 0 && nb >= 0, "negative size");
    if (na > kNoAllocMaxRows || nb > kNoAllocMaxRows) {
        set_error("invalid argument: na=%d, nb=%d exceeds the %d-row limit of the allocation-free matcher "
                  "(use fsb_match_bf_d)", na, nb, kNoAllocMaxRows);
        return FSB_ERR_ARG;
    }
    FSB_ARG((na == 0 || (d_a && d_q && d_t)) && (nb == 0 || d_b), "null device array");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (na < 2 || nb < 2) {
        FSB_CUDA(cudaMemsetAsync(d_n, 0, sizeof(int32_t), s));
        return FSB_OK;
    }
    void* base = nullptr;
    FSB_TRY(noalloc_scratch(&base));
    unsigned long long* key = static_cast<unsigned long long*>(base);
    Top2* part = reinterpret_cast<Top2*>(key + kNoAllocMaxRows);
    // the allocating matcher's plan, bounded by the top-2 table's capacity
    const BfPlan pl = bf_plan(&na, &nb, 1, kNoAllocSplitRows);
    BfPair one{d_a, d_b, part, key, d_q, d_t, d_n, na, nb};
    bf_place(pl, one, 0);
    FSB_CUDA(cudaMemsetAsync(key, 0xff, (size_t)nb * 8, s));
    FSB_TRY(launch_bf(pl, one, nullptr, 1, s));
    k_bf_merge<<<blocks(na, 256), 256, 0, s>>>(one, nullptr, ratio);
    k_unique_compact<<<1, COMPACT_T, 0, s>>>(key, nb, d_q, d_t, d_n);
    note_launch(2);
    FSB_CUDA(cudaGetLastError());
    return FSB_OK;
}
