// Device kernels of the Bine engine (sm_100a).
//
// All collectives here move or add whole rows of P virtual ranks that live
// in one HBM: the work is streaming integer/float traffic, bound by HBM
// bandwidth, so the kernels are built around 16-byte vector loads and
// stores, enough independent loads in flight per thread to cover DRAM
// latency (8 ranks per batch), streaming cache hints, and grids sized to the
// 148 SMs.  Nothing here is a dense contraction, so there are no tensor-core
// paths.
//
//   k_sum_*      fused reductions (allreduce, reduce_scatter, reduce): each
//                column of the P inputs is read once and the result written
//                once per destination; integer sums wrap exactly, the FAST
//                float order accumulates in FP64.
//   k_tree_*     fused reductions in the reference's exact float order: each
//                output segment carries the postfix program of its addition
//                tree (produced by the host planner), evaluated per column
//                with an in-register top of stack.
//   k_copy_*,    allgather, bcast, alltoall, scatter and gather as one pass of
//   k_spread     16-byte copies (one load, one or P stores).
//   k_steps      the reference's schedule executed level by level in one
//                cooperative launch, with a bounded grid-wide barrier between
//                levels that reports a timeout instead of hanging.
//   k_flow       the same schedule as a dataflow of segments: each starts
//                when the segments it reads and overwrites are done (bounded
//                waits on per-segment completion flags), so steps overlap.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace bine {
namespace dev {

constexpr int kThreads = 256;
constexpr int kMaxTreeDepth = 24;

// ---------------------------------------------------------------- memory
__device__ __forceinline__ uint4 ld_stream(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
// L2-coherent load (bypasses L1): rows written by other blocks earlier in
// the same launch must not be served from a stale L1 line.
__device__ __forceinline__ uint4 ld_plain(const void* p) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void st_stream(void* p, uint4 v) {
    asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                 : "memory");
}

// Strided lane vectors, for rows that do not share a 16-byte grid (packed
// rows of odd length, blocks of odd length): the 16 / sizeof(T) elements of
// a lane lie `STEP` elements apart and consecutive lanes hold consecutive
// elements, so every access of a warp is runs of min(32, STEP) elements
// wherever the row starts, and the vector arithmetic stays that of the 16-byte
// form.
// `n` elements of the vector exist (the first ones); the others read as 0.
template <typename T>
__device__ __forceinline__ T ld_stream_elem(const void* p) {
    T v;
    if constexpr (sizeof(T) == 8) {
        unsigned long long r;
        asm volatile("ld.global.nc.L1::no_allocate.u64 %0, [%1];" : "=l"(r) : "l"(p));
        memcpy(&v, &r, 8);
    } else if constexpr (sizeof(T) == 4) {
        unsigned r;
        asm volatile("ld.global.nc.L1::no_allocate.u32 %0, [%1];" : "=r"(r) : "l"(p));
        memcpy(&v, &r, 4);
    } else if constexpr (sizeof(T) == 2) {
        unsigned short r;
        asm volatile("ld.global.nc.L1::no_allocate.u16 %0, [%1];" : "=h"(r) : "l"(p));
        memcpy(&v, &r, 2);
    } else {
        unsigned r;
        asm volatile("ld.global.nc.L1::no_allocate.u8 %0, [%1];" : "=r"(r) : "l"(p));
        v = (T)r;
    }
    return v;
}
__device__ __forceinline__ uint4 ld_unit(const uint4* p) { return ld_stream(p); }
template <typename U>
__device__ __forceinline__ U ld_unit(const U* p) {
    return __ldg(p);  // through L1: neighbouring runs off the 128-byte grid share sectors
}
template <typename T, int STEP>
__device__ __forceinline__ uint4 ld_strided(const char* p, int n) {
    constexpr int N = 16 / sizeof(T);
    uint4 raw;
    T* t = reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int i = 0; i < N; i++) t[i] = i < n ? ld_stream_elem<T>(p + i * STEP * (int)sizeof(T)) : (T)0;
    return raw;
}
template <typename T>
__device__ __forceinline__ void st_cs(T* p, T v) {
    if constexpr (sizeof(T) == 16) st_stream(p, v);
    else __stcs(p, v);
}
template <typename T, int STEP>
__device__ __forceinline__ void st_strided(char* p, uint4 raw, int n) {
    constexpr int N = 16 / sizeof(T);
    const T* t = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < N; i++)
        if (i < n) __stcs(reinterpret_cast<T*>(p) + i * STEP, t[i]);
}

// ----------------------------------------------------------- lane algebra
// Accumulators: wrapping integers of the element type, FP64 for the FAST
// float order, the element type itself for the exact float order.
template <typename T>
struct AccOf {
    using type = T;
};
template <>
struct AccOf<float> {
    using type = double;
};

template <typename T>
__device__ __forceinline__ T add_exact(T a, T b) {
    return (T)(a + b);
}
template <>
__device__ __forceinline__ float add_exact<float>(float a, float b) {
    return __fadd_rn(a, b);
}
template <>
__device__ __forceinline__ double add_exact<double>(double a, double b) {
    return __dadd_rn(a, b);
}

template <typename T, typename A>
struct Lanes {
    static constexpr int N = 16 / sizeof(T);
    A v[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = (A)0;
    }
    __device__ __forceinline__ void add(uint4 raw) {
        const T* t = reinterpret_cast<const T*>(&raw);
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = add_exact<A>(v[i], (A)t[i]);
    }
    __device__ __forceinline__ uint4 pack() const {
        uint4 raw;
        T* t = reinterpret_cast<T*>(&raw);
#pragma unroll
        for (int i = 0; i < N; i++) t[i] = (T)v[i];
        return raw;
    }
};

template <typename T>
__device__ __forceinline__ uint4 vadd(uint4 a, uint4 b) {
    uint4 r;
    const T* x = reinterpret_cast<const T*>(&a);
    const T* y = reinterpret_cast<const T*>(&b);
    T* z = reinterpret_cast<T*>(&r);
#pragma unroll
    for (int i = 0; i < (int)(16 / sizeof(T)); i++) z[i] = add_exact<T>(x[i], y[i]);
    return r;
}

// ------------------------------------------------------- fused reductions
enum SumMode { kSumAllreduce = 0, kSumReduceScatter = 1, kSumReduce = 2 };

// Column sums.  A block owns tiles of COLS lane vectors at a time; its 256
// threads form 256/COLS row groups that split the P rows of a tile (group g
// sums rows [g*P/G, (g+1)*P/G) of its lane's vector, 8 loads in flight per
// thread), the partial sums meet in shared memory, and all threads then
// store the result rows.  The host picks COLS (64 vectors and 4 row groups;
// one group below P = 16; narrower tiles for calls too small to give every
// SM two tiles) and launches one block per tile up to 64 blocks per SM,
// beyond which blocks walk the tiles grid-stride.
//
// The call covers elements [0, n) of rows that start at `in` and `out`;
// reduce_scatter: `blk` elements per destination rank, and `in` is element
// `e0` of the row.  VEC: lane vectors of 16 contiguous, aligned bytes (n is
// whole vectors, blk counts vectors, e0 is 0; with blk in elements int8 at P =
// 768 and 16 elements took 7.6 us, 6.5 so).  Otherwise strided ones
// (ld_strided, COLS elements apart), for rows off the 16-byte grid and for the
// last partial vector, except for few ranks: the loop over the rows is the
// same, with four loads of 4 bytes in the place of one of 16, bound by their
// issue.  They replaced one thread per element with its P rows in a chain
// (int32 allreduce, us per call): P = 96 at 262,147 elements per rank 47.7 ->
// 39.3 (37.3 at 262,144, on the grid), P = 256 at 1,048,577 509 -> 381, P =
// 300 at 777 int64 28.3 -> 8.1, P = 500 at 1 15.0 -> 7.3.
constexpr int kSumCols = 8;  // the narrowest tile (32 row groups)

template <typename T, int MODE, int COLS, bool VEC>
__global__ void __launch_bounds__(kThreads) k_sum_vec(const char* __restrict__ in, long long in_stride,
                                                      char* __restrict__ out, long long out_stride, int P,
                                                      long long n, long long blk, int root, long long e0) {
    using A = typename AccOf<T>::type;
    constexpr int G = kThreads / COLS;
    constexpr int L = 16 / sizeof(T);
    __shared__ Lanes<T, A> part[G][COLS];
    __shared__ uint4 res[COLS];
    const int lane = threadIdx.x % COLS, grp = threadIdx.x / COLS;
    const int per = (P + G - 1) / G;
    const int r0 = min(P, grp * per), r1 = min(P, r0 + per);
    const long long ntiles = (n + COLS * L - 1) / (COLS * L);
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // The lane's vector: first element, and how many of its elements exist.
        const long long e = tile * (COLS * L) + (VEC ? lane * L : lane);
        const int have = VEC ? (e < n ? L : 0) : (int)max(0ll, min((long long)L, (n - e + COLS - 1) / COLS));
        const auto ld = [&](const char* p) { return VEC ? ld_stream(p) : ld_strided<T, COLS>(p, have); };
        Lanes<T, A> acc;
        acc.zero();
        if (have > 0) {
            const char* p = in + e * (long long)sizeof(T);
            int r = r0;
            for (; r + 8 <= r1; r += 8) {
                uint4 v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = ld(p + (long long)(r + u) * in_stride);
#pragma unroll
                for (int u = 0; u < 8; u++) acc.add(v[u]);
            }
            for (; r < r1; r++) acc.add(ld(p + (long long)r * in_stride));
        }
        if (G > 1) {
            part[grp][lane] = acc;
            __syncthreads();
            if (grp == 0) {
                Lanes<T, A> sum = part[0][lane];
#pragma unroll
                for (int g = 1; g < G; g++)
#pragma unroll
                    for (int i = 0; i < Lanes<T, A>::N; i++) sum.v[i] = add_exact<A>(sum.v[i], part[g][lane].v[i]);
                res[lane] = sum.pack();
            }
            __syncthreads();
        } else {
            res[lane] = acc.pack();
        }
        if (have > 0) {
            const uint4 v = res[lane];
            const auto st = [&](char* q) {
                if (VEC) st_stream(q, v);
                else st_strided<T, COLS>(q, v, have);
            };
            if (MODE == kSumAllreduce) {
                char* q = out + e * (long long)sizeof(T);
                for (int d = grp; d < P; d += G) st(q + (long long)d * out_stride);
            } else if (grp == 0) {
                if (MODE == kSumReduce) {
                    st(out + (long long)root * out_stride + e * (long long)sizeof(T));
                } else if (VEC) {
                    const long long col = tile * COLS + lane, owner = col / blk;
                    st(out + owner * out_stride + (col - owner * blk) * 16);
                } else {
                    const T* t = reinterpret_cast<const T*>(&v);
#pragma unroll
                    for (int i = 0; i < L; i++) {
                        if (i < have) {
                            const long long x = e0 + e + (long long)i * COLS, owner = x / blk;
                            __stcs(reinterpret_cast<T*>(out + owner * out_stride) + (x - owner * blk), t[i]);
                        }
                    }
                }
            }
        }
        if (G > 1) __syncthreads();
    }
}

// Sums off the 16-byte grid of 1-byte elements and of few ranks, elements [e0,
// e0 + n) of every row, one per thread: a strided lane vector of bytes would
// take 16 loads of one byte each (int8 allreduce at P = 96, 262,147 elements
// per rank: 20.7 us here, 33.3 us strided), and with few rows one thread's
// loads are few.  reduce_scatter: `blk` elements per rank.
constexpr int kSumManyElems = 65536;  // from here on few ranks are up to 24 or 40 (launch_sum)
template <typename T, int MODE>
__global__ void __launch_bounds__(kThreads) k_sum_scalar(const char* __restrict__ in, long long in_stride,
                                                         char* __restrict__ out, long long out_stride, int P,
                                                         long long e0, long long n, long long blk, int root) {
    using A = typename AccOf<T>::type;
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const long long e = e0 + i;
        A acc = (A)0;
        for (int r = 0; r < P; r++) acc = add_exact<A>(acc, (A) * (const T*)(in + (long long)r * in_stride + e * sizeof(T)));
        const T res = (T)acc;
        if (MODE == kSumAllreduce) {
            for (int d = 0; d < P; d++) *(T*)(out + (long long)d * out_stride + e * sizeof(T)) = res;
        } else if (MODE == kSumReduceScatter) {
            long long owner = e / blk;
            *(T*)(out + owner * out_stride + (e - owner * blk) * sizeof(T)) = res;
        } else {
            *(T*)(out + (long long)root * out_stride + e * sizeof(T)) = res;
        }
    }
}

// ------------------------------------------- fused reductions, exact order
struct TreeEntry {  // one postfix entry: push input (rank, out + shift), then `adds` additions
    int32_t rank;
    int32_t adds;
    int64_t shift;
};
struct TreeSeg {  // output elements [off, off + n) of `rank` (-1: all ranks)
    int64_t off, n;
    int32_t rank, prog_begin, prog_len, depth;
};
struct TreeTile {  // `n` elements starting `start` elements into segment `seg`
    int32_t seg, pad;
    int64_t start, n;
};

// Evaluation stack of a postfix program (the entries below the top, which
// stays in registers).  SMEM: in the block's dynamic shared memory, slot j
// of thread t at base[j * kThreads + t], so a warp's 16-byte accesses fall
// on consecutive words; sized by the host to the programs' Sethi-Ullman
// depth.  Otherwise a local array (deep programs only): its indexing is
// dynamic, so it lives in local memory and its traffic reaches L2.
template <bool SMEM>
struct EvalStack;
template <>
struct EvalStack<true> {
    uint4* base;
    __device__ __forceinline__ void init(uint4* smem_stack) { base = smem_stack + threadIdx.x; }
    __device__ __forceinline__ void set(int j, uint4 v) { base[j * kThreads] = v; }
    __device__ __forceinline__ uint4 get(int j) const { return base[j * kThreads]; }
};
template <>
struct EvalStack<false> {
    uint4 a[kMaxTreeDepth];
    __device__ __forceinline__ void init(uint4*) {}
    __device__ __forceinline__ void set(int j, uint4 v) { a[j] = v; }
    __device__ __forceinline__ uint4 get(int j) const { return a[j]; }
};

// Vector form: every shift and offset is a multiple of 16 bytes.  One tile
// per block; each thread owns one 16-byte column of the tile.
template <typename T, bool SMEM>
__global__ void __launch_bounds__(kThreads) k_tree_vec(const char* __restrict__ in, long long in_stride,
                                                       char* __restrict__ out, long long out_stride, int P,
                                                       const TreeSeg* __restrict__ segs,
                                                       const TreeEntry* __restrict__ prog,
                                                       const TreeTile* __restrict__ tiles, int ntiles,
                                                       int stack_off) {
    extern __shared__ uint4 sdyn[];
    TreeEntry* sprog = reinterpret_cast<TreeEntry*>(sdyn);
    EvalStack<SMEM> stk;
    stk.init(sdyn + stack_off);
    constexpr int L = 16 / sizeof(T);
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const TreeTile tile = tiles[t];
        const TreeSeg sg = segs[tile.seg];
        __syncthreads();
        // Staged with each leaf's byte offset (rank row + shift) precomputed.
        for (int i = threadIdx.x; i < sg.prog_len; i += blockDim.x) {
            TreeEntry q = prog[sg.prog_begin + i];
            q.shift = (long long)q.rank * in_stride + q.shift * (long long)sizeof(T);
            sprog[i] = q;
        }
        __syncthreads();
        const long long col = (long long)threadIdx.x * L;
        if (col >= tile.n) continue;
        const long long e = sg.off + tile.start + col;  // output element
        const char* base = in + e * (long long)sizeof(T);
        uint4 top = make_uint4(0, 0, 0, 0);
        int sp = 0;
        const int len = sg.prog_len;
        // Loads run 8 entries ahead of the additions.
        uint4 ring[8];
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (u < len) {
                const TreeEntry q = sprog[u];
                ring[u] = ld_stream(base + q.shift);
            }
        for (int k0 = 0; k0 < len; k0 += 8) {
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int k = k0 + u;
                if (k < len) {
                    const uint4 v = ring[u];
                    if (k + 8 < len) {
                        const TreeEntry q = sprog[k + 8];
                        ring[u] = ld_stream(base + q.shift);
                    }
                    if (k > 0) stk.set(sp++, top);
                    top = v;
                    for (int a = sprog[k].adds; a > 0; a--) top = vadd<T>(stk.get(--sp), top);
                }
            }
        }
        if (sg.rank < 0) {
            for (int d = 0; d < P; d++) st_stream(out + (long long)d * out_stride + e * (long long)sizeof(T), top);
        } else {
            st_stream(out + (long long)sg.rank * out_stride + e * (long long)sizeof(T), top);
        }
    }
}

// Split form of k_tree_vec.  The host cut every segment's addition tree
// into `nparts` disjoint subtrees (the "parts", left to right; K of them,
// or 2K when that balances the warps better) and a combine program whose
// leaves are the parts, and assigned the parts to K warps longest first, so
// the warps carry near-equal numbers of leaves even when the tree is
// unbalanced (non-power-of-two P).  A block of 8 warps owns 8/K
// column groups of 32 vectors; warp w evaluates its parts for group w / K,
// one vector per lane, so every load of a warp is 512 contiguous bytes of
// one rank row (as in k_sum_vec).  The partial sums meet in shared memory;
// each warp then runs the combine program for its group's 32 vectors and
// stores every K-th destination row.  The additions and their association
// are exactly the tree's.  Shorter tasks remove the tail of the last wave
// when the output has few vectors per resident thread.
struct TreeComb {  // combine entry: push part `part`, then `adds` additions
    int32_t part, adds;
};

// Evaluates program entries [b, b + len) for one lane vector; `ld` loads it
// at a leaf's byte offset (entries hold it precomputed), kRing entries ahead
// of the additions.
template <typename T, bool SMEM, int kRing, typename Ld>
__device__ __forceinline__ uint4 eval_program(const Ld& ld, const TreeEntry* sprog, int b, int len,
                                              EvalStack<SMEM>& stk) {
    uint4 top = make_uint4(0, 0, 0, 0);
    int sp = 0;
    uint4 ring[kRing];
#pragma unroll
    for (int u = 0; u < kRing; u++)
        if (u < len) {
            const TreeEntry q = sprog[b + u];
            ring[u] = ld(q.shift);
        }
    for (int k0 = 0; k0 < len; k0 += kRing) {
#pragma unroll
        for (int u = 0; u < kRing; u++) {
            const int k = k0 + u;
            if (k < len) {
                const uint4 v = ring[u];
                if (k + kRing < len) {
                    const TreeEntry q = sprog[b + k + kRing];
                    ring[u] = ld(q.shift);
                }
                if (k > 0) stk.set(sp++, top);
                top = v;
                for (int a = sprog[b + k].adds; a > 0; a--) top = vadd<T>(stk.get(--sp), top);
            }
        }
    }
    return top;
}

template <typename T, int K, bool SMEM>
__global__ void __launch_bounds__(kThreads) k_tree_split(const char* __restrict__ in, long long in_stride,
                                                         char* __restrict__ out, long long out_stride, int P,
                                                         const TreeSeg* __restrict__ segs,
                                                         const TreeEntry* __restrict__ prog,
                                                         const int* __restrict__ parts,
                                                         const TreeComb* __restrict__ comb,
                                                         const int* __restrict__ assign,
                                                         const TreeTile* __restrict__ tiles, int ntiles,
                                                         int nparts, int stack_off) {
    extern __shared__ uint4 sdyn[];
    TreeEntry* sprog = reinterpret_cast<TreeEntry*>(sdyn);
    EvalStack<SMEM> stk;
    stk.init(sdyn + stack_off);
    constexpr int kWarps = kThreads / 32;
    constexpr int kGroups = kWarps / K;
    constexpr int KP = 2 * K;
    // Per segment: part offsets, combine program, and the parts of each warp
    // (nparts <= KP part indices ordered by warp, then K + 1 offsets).
    __shared__ int spart[KP + 1];
    __shared__ TreeComb scomb[KP];
    __shared__ int sasg[KP + K + 1];
    __shared__ uint4 partial[kGroups][KP][32];
    constexpr int L = 16 / sizeof(T);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = warp % K, g = warp / K;
    int cur = -1;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const TreeTile tile = tiles[t];
        const TreeSeg sg = segs[tile.seg];
        __syncthreads();  // the previous tile's partials and program are consumed
        if (tile.seg != cur) {  // block-uniform
            for (int i = threadIdx.x; i < sg.prog_len; i += blockDim.x) {
                TreeEntry q = prog[sg.prog_begin + i];
                q.shift = (long long)q.rank * in_stride + q.shift * (long long)sizeof(T);  // byte offset
                sprog[i] = q;
            }
            if (threadIdx.x <= nparts) spart[threadIdx.x] = parts[(long long)tile.seg * (nparts + 1) + threadIdx.x];
            if (threadIdx.x < nparts) scomb[threadIdx.x] = comb[(long long)tile.seg * nparts + threadIdx.x];
            if (threadIdx.x < nparts + K + 1)
                sasg[threadIdx.x] = assign[(long long)tile.seg * (nparts + K + 1) + threadIdx.x];
            __syncthreads();
            cur = tile.seg;
        }
        const long long col = (long long)(g * 32 + lane) * L;
        const bool active = col < tile.n;
        const long long e = sg.off + tile.start + col;
        if (active) {
            for (int pi = sasg[nparts + j]; pi < sasg[nparts + j + 1]; pi++) {
                const int p = sasg[pi];
                const char* base = in + e * (long long)sizeof(T);
                partial[g][p][lane] = eval_program<T, SMEM, 4>([&](long long off) { return ld_stream(base + off); },
                                                               sprog, spart[p], spart[p + 1] - spart[p], stk);
            }
        }
        __syncthreads();
        if (!active) continue;
        uint4 top = make_uint4(0, 0, 0, 0);
        int csp = 0;  // the parts' stack is empty again: the combine reuses it
        for (int q = 0; q < nparts; q++) {
            const TreeComb c = scomb[q];
            if (q > 0) stk.set(csp++, top);
            top = partial[g][c.part][lane];
            for (int a = c.adds; a > 0; a--) top = vadd<T>(stk.get(--csp), top);
        }
        if (sg.rank < 0) {
            for (int d = j; d < P; d += K) st_stream(out + (long long)d * out_stride + e * (long long)sizeof(T), top);
        } else if (j == 0) {
            st_stream(out + (long long)sg.rank * out_stride + e * (long long)sizeof(T), top);
        }
    }
}

// Row-aligned form of k_tree_split, for calls whose trees have few
// shapes.  In allreduce every leaf reads its rank's row at the output's own
// column, and the segments' trees (one segment per block of the
// reference's vector) share one shape, or a few (at most kFlatShapes):
// segments of one shape differ only in the order of their ranks.  The tiles of k_tree_split start at each segment's
// first 16-byte boundary; with non-power-of-two P that is an arbitrary
// 16-byte offset, so every 512-byte warp access straddles five 128-byte
// lines, and a segment's last tile is mostly empty.  Here tiles follow the
// output row's own grid of 32-vector groups instead: `tile.start` is a
// multiple of the tile width (in elements, from the row start), a tile may
// hold the ends of several segments of one shape (`tile.pad & 0xff` of them
// from `tile.seg`, in the order of their bodies; the shape is
// `tile.pad >> 8`, and the block stages that shape's plan when it changes),
// and each lane evaluates its own segment's ranks.  Where segments of
// several shapes meet in one tile's columns, each shape has its own tile
// there, and lanes whose vector belongs to another shape idle.
//
// A vector that straddles two consecutive segments (an "edge": its first
// `cut` elements end segment q, the rest begin segment q + 1) is evaluated
// by k_tree_edges, beside this kernel, as a whole 16-byte vector, instead of
// element by element.  The additions, and so the results, are exactly the
// trees'.
//
//   body[2q], body[2q+1] segment q's vector body [lo, hi), in elements
//   ranks[q * pitch + k] the rank of entry k of segment q's split program;
//   ranks_t[k * nq + q] the same, entry-major (edge lanes read consecutive q)
//   adds[h * len + k]   additions after entry k of shape h's programs
//   parts, comb, assign shape h's split plan (as in k_tree_split), at
//                       h * (nparts + 1), h * nparts, h * (nparts + K + 1)
constexpr int kFlatSegs = 8;    // segments one row tile may touch
constexpr int kFlatShapes = 8;  // tree shapes one call may have

struct FlatEdge {  // the vector at element `e`: elements [e, e + cut) in segment q, the rest in q + 1
    int64_t e;
    int32_t q, cut;
};

struct FlatArgs {
    const char* in;
    long long in_stride;
    char* out;
    long long out_stride;
    int P;
    const int64_t* body;
    const uint16_t* ranks;
    const uint16_t* ranks_t;
    int pitch, nq;
    const uint8_t* adds;
    int len;  // bytes of `adds`, a multiple of 16
    const int* parts;
    const TreeComb* comb;
    const int* assign;
    const FlatEdge* edges;
    const uint8_t* shape;  // edges: the tree shape of each segment (row order)
    int nshape;
    const TreeTile* tiles;
    int ntiles, nparts;
    int ranks_off, stack_off;  // dynamic shared memory offsets, in 16-byte words
};

// Evaluates entries [b, b + len) of a program whose additions are
// `adds[k]` and whose ranks are `rk[k]` (a row of the shared-memory rank
// table), for one 16-byte vector at `base`; loads run kRing entries ahead
// of the additions.
template <typename T, bool SMEM, int kRing>
__device__ __forceinline__ uint4 eval_ranks(const char* __restrict__ base, long long stride, const uint16_t* rk,
                                            const uint8_t* adds, int b, int len, EvalStack<SMEM>& stk) {
    uint4 top = make_uint4(0, 0, 0, 0);
    int sp = 0;
    uint4 ring[kRing];
#pragma unroll
    for (int u = 0; u < kRing; u++)
        if (u < len) ring[u] = ld_stream(base + (long long)rk[b + u] * stride);
    for (int k0 = 0; k0 < len; k0 += kRing) {
#pragma unroll
        for (int u = 0; u < kRing; u++) {
            const int k = k0 + u;
            if (k < len) {
                const uint4 v = ring[u];
                if (k + kRing < len) ring[u] = ld_stream(base + (long long)rk[b + k + kRing] * stride);
                if (k > 0) stk.set(sp++, top);
                top = v;
                for (int a = adds[b + k]; a > 0; a--) top = vadd<T>(stk.get(--sp), top);
            }
        }
    }
    return top;
}

template <typename T, int K, bool SMEM>
__global__ void __launch_bounds__(kThreads) k_tree_flat(const FlatArgs A) {
    extern __shared__ uint4 sdyn[];
    uint8_t* sadds = reinterpret_cast<uint8_t*>(sdyn);
    uint16_t* sranks = reinterpret_cast<uint16_t*>(sdyn + A.ranks_off);
    EvalStack<SMEM> stk;
    stk.init(sdyn + A.stack_off);
    constexpr int kWarps = kThreads / 32;
    constexpr int kGroups = kWarps / K;
    constexpr int KP = 2 * K;
    __shared__ int spart[KP + 1];
    __shared__ TreeComb scomb[KP];
    __shared__ int sasg[KP + K + 1];
    __shared__ int64_t slo[kFlatSegs], shi[kFlatSegs];
    __shared__ uint4 partial[kGroups][KP][32];
    constexpr int L = 16 / sizeof(T);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = warp % K, g = warp / K;
    const int nparts = A.nparts;
    const int words = A.pitch / 8;  // 16-byte words of one segment's ranks
    const uint4* granks = reinterpret_cast<const uint4*>(A.ranks);
    uint4* sranks4 = reinterpret_cast<uint4*>(sranks);
    int cur = -1;  // the tree shape whose plan is staged
    for (int t = blockIdx.x; t < A.ntiles; t += gridDim.x) {
        const TreeTile tile = A.tiles[t];
        const int s0 = tile.seg, ns = tile.pad & 0xff, shape = tile.pad >> 8;
        __syncthreads();  // the previous tile's partials, ranks and plan are consumed
        if (shape != cur) {  // block-uniform: the plan of this tile's tree shape
            const uint4* ga = reinterpret_cast<const uint4*>(A.adds + (long long)shape * A.len);
            for (int i = threadIdx.x; i < A.len / 16; i += blockDim.x) sdyn[i] = ga[i];
            if (threadIdx.x <= nparts) spart[threadIdx.x] = A.parts[shape * (nparts + 1) + threadIdx.x];
            if (threadIdx.x < nparts) scomb[threadIdx.x] = A.comb[shape * nparts + threadIdx.x];
            if (threadIdx.x < nparts + K + 1) sasg[threadIdx.x] = A.assign[shape * (nparts + K + 1) + threadIdx.x];
            cur = shape;
        }
        for (int i = threadIdx.x; i < ns * words; i += blockDim.x) sranks4[i] = granks[(long long)s0 * words + i];
        if (threadIdx.x < ns) {
            slo[threadIdx.x] = A.body[2 * (s0 + threadIdx.x)];
            shi[threadIdx.x] = A.body[2 * (s0 + threadIdx.x) + 1];
        }
        __syncthreads();
        const long long e = tile.start + (long long)(g * 32 + lane) * L;  // first element of the lane's vector
        int slot = -1;
        if (e < tile.start + tile.n)
            for (int q = 0; q < ns; q++)
                if (e >= slo[q] && e < shi[q]) slot = q;
        const bool active = slot >= 0;
        if (active) {
            const uint16_t* rk = sranks + slot * A.pitch;
            for (int pi = sasg[nparts + j]; pi < sasg[nparts + j + 1]; pi++) {
                const int p = sasg[pi];
                partial[g][p][lane] = eval_ranks<T, SMEM, 4>(A.in + e * (long long)sizeof(T), A.in_stride, rk,
                                                             sadds, spart[p], spart[p + 1] - spart[p], stk);
            }
        }
        __syncthreads();
        if (!active) continue;
        uint4 top = make_uint4(0, 0, 0, 0);
        int csp = 0;
        for (int q = 0; q < nparts; q++) {
            const TreeComb c = scomb[q];
            if (q > 0) stk.set(csp++, top);
            top = partial[g][c.part][lane];
            for (int a = c.adds; a > 0; a--) top = vadd<T>(stk.get(--csp), top);
        }
        for (int d = j; d < A.P; d += K)
            st_stream(A.out + (long long)d * A.out_stride + e * (long long)sizeof(T), top);
    }
}

// Edge form of eval_ranks: the ranks come from the entry-major global
// table (`rt` at the lane's segment; entry k at rt[k * nq]) and are read
// one ring ahead of the loads that use them, so that a rank's L2 latency is
// not added to every leaf's.
template <typename T, bool SMEM, int kRing>
__device__ __forceinline__ uint4 eval_edge(const char* __restrict__ base, long long stride,
                                           const uint16_t* __restrict__ rt, int nq, const uint8_t* adds, int b,
                                           int len, EvalStack<SMEM>& stk) {
    uint4 top = make_uint4(0, 0, 0, 0);
    int sp = 0;
    uint4 ring[kRing];
    int rr[kRing];
#pragma unroll
    for (int u = 0; u < kRing; u++)
        if (u < len) rr[u] = __ldg(rt + (long long)(b + u) * nq);
#pragma unroll
    for (int u = 0; u < kRing; u++)
        if (u < len) {
            ring[u] = ld_stream(base + (long long)rr[u] * stride);
            if (u + kRing < len) rr[u] = __ldg(rt + (long long)(b + u + kRing) * nq);
        }
    for (int k0 = 0; k0 < len; k0 += kRing) {
#pragma unroll
        for (int u = 0; u < kRing; u++) {
            const int k = k0 + u;
            if (k < len) {
                const uint4 v = ring[u];
                if (k + kRing < len) {
                    ring[u] = ld_stream(base + (long long)rr[u] * stride);
                    if (k + 2 * kRing < len) rr[u] = __ldg(rt + (long long)(b + k + 2 * kRing) * nq);
                }
                if (k > 0) stk.set(sp++, top);
                top = v;
                for (int a = adds[b + k]; a > 0; a--) top = vadd<T>(stk.get(--sp), top);
            }
        }
    }
    return top;
}

// The edges of the row-aligned form (see above).  Their trees are cut into
// kEdgeParts subtrees of their own (the edge split plan of each shape h:
// `parts` at h * (kEdgeParts + 1), `comb` at h * kEdgeParts, `adds` at
// h * len; ranks_t in that plan's entry order, and `shape` giving each
// segment's shape), so that an edge's critical path is P / kEdgeParts
// leaves whatever the row tiles' split.
// Block b owns edges [32 * (b / 2), +32) and segment side b % 2 (0: the
// segment the edge vector ends, 1: the one it starts); warp w evaluates
// part w for its lane's edge, the partial sums meet in shared memory, and
// every lane combines them and stores the elements of its side (the first
// `cut` elements of the vector, or the rest) to the rows w, w + 8, ...  The
// two sides of an edge run in neighbouring blocks, so the two halves of its
// 16-byte vector reach L2 close together.
constexpr int kEdgeParts = 8;

template <typename T, bool SMEM>
__global__ void __launch_bounds__(kThreads) k_tree_edges(const FlatArgs A, int nedges) {
    extern __shared__ uint4 sdyn[];
    uint8_t* sadds = reinterpret_cast<uint8_t*>(sdyn);
    EvalStack<SMEM> stk;
    stk.init(sdyn + A.stack_off);
    static_assert(kThreads / 32 == kEdgeParts, "one warp per edge part");
    // The edge plans of every tree shape (a lane's edge may end a segment
    // of one shape and begin one of another).
    __shared__ int spart[kFlatShapes][kEdgeParts + 1];
    __shared__ TreeComb scomb[kFlatShapes][kEdgeParts];
    __shared__ uint4 partial[kEdgeParts][32];
    constexpr int L = 16 / sizeof(T);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < A.nshape * A.len / 16; i += blockDim.x)
        sdyn[i] = reinterpret_cast<const uint4*>(A.adds)[i];
    for (int i = threadIdx.x; i < A.nshape * (kEdgeParts + 1); i += blockDim.x)
        spart[i / (kEdgeParts + 1)][i % (kEdgeParts + 1)] = A.parts[i];
    for (int i = threadIdx.x; i < A.nshape * kEdgeParts; i += blockDim.x)
        scomb[i / kEdgeParts][i % kEdgeParts] = A.comb[i];
    const int ngroups = (nedges + 31) / 32;
    for (int t = blockIdx.x; t < 2 * ngroups; t += gridDim.x) {
        const int side = t & 1, ei = (t >> 1) * 32 + lane;
        const bool act = ei < nedges;
        FlatEdge ed{0, 0, 0};
        int sh = 0;
        if (act) {
            ed = A.edges[ei];
            sh = A.shape[ed.q + side];
        }
        __syncthreads();  // the previous partials are consumed (and the plans staged)
        if (act)
            partial[w][lane] = eval_edge<T, SMEM, 8>(A.in + ed.e * (long long)sizeof(T), A.in_stride,
                                                     A.ranks_t + ed.q + side, A.nq, sadds + sh * A.len, spart[sh][w],
                                                     spart[sh][w + 1] - spart[sh][w], stk);
        __syncthreads();
        if (!act) continue;
        uint4 top = make_uint4(0, 0, 0, 0);
        int csp = 0;
        for (int q = 0; q < kEdgeParts; q++) {
            const TreeComb c = scomb[sh][q];
            if (q > 0) stk.set(csp++, top);
            top = partial[c.part][lane];
            for (int a = c.adds; a > 0; a--) top = vadd<T>(stk.get(--csp), top);
        }
        const T* r = reinterpret_cast<const T*>(&top);
        const int x0 = side ? ed.cut : 0, x1 = side ? L : ed.cut;
        for (int d = w; d < A.P; d += kEdgeParts) {
            T* o = reinterpret_cast<T*>(A.out + (long long)d * A.out_stride + ed.e * (long long)sizeof(T));
            for (int x = x0; x < x1; x++) o[x] = r[x];
        }
    }
}

// Element form for the short head and tail pieces of segments (fewer
// elements than one 16-byte vector).  Per tile the block
//   1. loads every leaf value of the tile's elements into shared memory in
//      one parallel round;
//   2. evaluates the tree's parts (the split plan's `nparts` subtrees, or
//      the whole tree as one part) with one thread per (element, part);
//   3. combines each element's partials in the tree's order;
//   4. spreads the P destination stores over all its threads.
// Without steps 2 and 4 one thread per element ran the whole P-leaf
// program and issued all P stores, which made this small kernel as long as
// the vector kernel beside it at P = 1000.
constexpr int kMaxParts = 16;
constexpr int kMaxPiece = 4;  // elements of a piece: fewer than one vector

template <typename T>
__global__ void __launch_bounds__(kThreads) k_tree_staged(const char* __restrict__ in, long long in_stride,
                                                          char* __restrict__ out, long long out_stride, int P,
                                                          const TreeSeg* __restrict__ segs,
                                                          const TreeEntry* __restrict__ prog,
                                                          const int* __restrict__ parts,
                                                          const TreeComb* __restrict__ comb, int nparts,
                                                          const TreeTile* __restrict__ tiles, int ntiles,
                                                          int vals_off) {
    extern __shared__ uint4 sdyn[];
    TreeEntry* sprog = reinterpret_cast<TreeEntry*>(sdyn);
    T* vals = reinterpret_cast<T*>(sdyn + vals_off);
    __shared__ int spart[kMaxParts + 1];
    __shared__ TreeComb scomb[kMaxParts];
    __shared__ T partial[kMaxPiece][kMaxParts];
    __shared__ T res[kMaxPiece];
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const TreeTile tile = tiles[t];
        const TreeSeg sg = segs[tile.seg];
        const int len = sg.prog_len, n = (int)tile.n;
        __syncthreads();  // the previous tile's values and results are consumed
        for (int i = threadIdx.x; i < len; i += blockDim.x) sprog[i] = prog[sg.prog_begin + i];
        if (threadIdx.x <= nparts) spart[threadIdx.x] = parts[(long long)tile.seg * (nparts + 1) + threadIdx.x];
        if (threadIdx.x < nparts) scomb[threadIdx.x] = comb[(long long)tile.seg * nparts + threadIdx.x];
        __syncthreads();
        const long long e0 = sg.off + tile.start;
        for (int i = threadIdx.x; i < n * len; i += blockDim.x) {
            const int jj = i / len, k = i - jj * len;
            const TreeEntry q = sprog[k];
            vals[i] = *(const T*)(in + (long long)q.rank * in_stride + (e0 + jj + q.shift) * (long long)sizeof(T));
        }
        __syncthreads();
        for (int w = threadIdx.x; w < n * nparts; w += blockDim.x) {
            const int jj = w / nparts, p = w - jj * nparts;
            const T* v = vals + jj * len;
            T stk[kMaxTreeDepth];
            T top = (T)0;
            int sp = 0;
            for (int k = spart[p]; k < spart[p + 1]; k++) {
                if (k > spart[p]) stk[sp++] = top;
                top = v[k];
                for (int a = sprog[k].adds; a > 0; a--) top = add_exact<T>(stk[--sp], top);
            }
            partial[jj][p] = top;
        }
        __syncthreads();
        if (threadIdx.x < n) {
            T stk[kMaxParts];
            T top = (T)0;
            int sp = 0;
            for (int q = 0; q < nparts; q++) {
                if (q > 0) stk[sp++] = top;
                top = partial[threadIdx.x][scomb[q].part];
                for (int a = scomb[q].adds; a > 0; a--) top = add_exact<T>(stk[--sp], top);
            }
            res[threadIdx.x] = top;
        }
        __syncthreads();
        if (sg.rank < 0) {
            for (int w = threadIdx.x; w < P * n; w += blockDim.x) {
                const int d = w / n, jj = w - d * n;
                *(T*)(out + (long long)d * out_stride + (e0 + jj) * (long long)sizeof(T)) = res[jj];
            }
        } else if (threadIdx.x < n) {
            *(T*)(out + (long long)sg.rank * out_stride + (e0 + threadIdx.x) * (long long)sizeof(T)) = res[threadIdx.x];
        }
    }
}

// Form for layouts and segments off the 16-byte grid (packed rows of odd
// length, blocks of odd length): k_tree_split over strided lane vectors.  A
// tile is up to (8 / K) groups of 32 lanes times 16 / sizeof(T) elements of
// one segment; element i of a lane's vector lies 32 * i elements after its
// first, so every load and store of a warp is one run of 32 elements.  K = 1
// evaluates whole programs (no split plan).
//
// The arithmetic per row is that of the aligned form, with four 4-byte loads
// in the place of one of 16: bound by the latency and the issue of those
// loads at four blocks of 64 registers per SM (42 % of the warps; float32 at
// P = 96, 262,147 elements: DRAM and L1 at 42 and 43 % of their peaks, 70 % of
// the copy rate; most stalled on loads in flight).  It replaced a kernel of
// one element per thread and one load in flight on 1,024-element tiles
// (288 blocks): float32 allreduce at P = 96, 262,147 elements per rank,
// 232 -> 44.3 us per call (867 -> 4,550 GB/s); P = 256 at 1,048,579
// elements runs at 5,180 GB/s, reduce_scatter at P = 64 and 32,769 at 5,530.
template <typename T, int K, bool SMEM>
__global__ void __launch_bounds__(kThreads) k_tree_strided(const char* __restrict__ in, long long in_stride,
                                                           char* __restrict__ out, long long out_stride, int P,
                                                           const TreeSeg* __restrict__ segs,
                                                           const TreeEntry* __restrict__ prog,
                                                           const int* __restrict__ parts,
                                                           const TreeComb* __restrict__ comb,
                                                           const int* __restrict__ assign,
                                                           const TreeTile* __restrict__ tiles, int ntiles,
                                                           int nparts, int stack_off) {
    extern __shared__ uint4 sdyn[];
    TreeEntry* sprog = reinterpret_cast<TreeEntry*>(sdyn);
    EvalStack<SMEM> stk;
    stk.init(sdyn + stack_off);
    constexpr int kWarps = kThreads / 32;
    constexpr int kGroups = kWarps / K;
    constexpr int KP = 2 * K;
    __shared__ int spart[KP + 1];
    __shared__ TreeComb scomb[KP];
    __shared__ int sasg[KP + K + 1];
    __shared__ uint4 partial[K > 1 ? kGroups : 1][K > 1 ? KP : 1][32];
    constexpr int L = 16 / sizeof(T);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = warp % K, g = warp / K;
    int cur = -1;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const TreeTile tile = tiles[t];
        const TreeSeg sg = segs[tile.seg];
        __syncthreads();  // the previous tile's partials and program are consumed
        if (tile.seg != cur) {  // block-uniform
            for (int i = threadIdx.x; i < sg.prog_len; i += blockDim.x) {
                TreeEntry q = prog[sg.prog_begin + i];
                q.shift = (long long)q.rank * in_stride + q.shift * (long long)sizeof(T);  // byte offset
                sprog[i] = q;
            }
            if constexpr (K > 1) {
                if (threadIdx.x <= nparts) spart[threadIdx.x] = parts[(long long)tile.seg * (nparts + 1) + threadIdx.x];
                if (threadIdx.x < nparts) scomb[threadIdx.x] = comb[(long long)tile.seg * nparts + threadIdx.x];
                if (threadIdx.x < nparts + K + 1)
                    sasg[threadIdx.x] = assign[(long long)tile.seg * (nparts + K + 1) + threadIdx.x];
            }
            __syncthreads();
            cur = tile.seg;
        }
        const long long col = (long long)g * (32 * L) + lane;  // first element of the lane's vector, in the tile
        const int nact = (int)min((long long)L, (tile.n - col + 31) / 32);  // its elements inside the tile
        const long long byte = (sg.off + tile.start + col) * (long long)sizeof(T);
        const char* base = in + byte;
        const auto ld = [&](long long off) { return ld_strided<T, 32>(base + off, nact); };
        uint4 top = make_uint4(0, 0, 0, 0);
        if constexpr (K > 1) {
            if (nact > 0) {
                for (int pi = sasg[nparts + j]; pi < sasg[nparts + j + 1]; pi++) {
                    const int p = sasg[pi];
                    partial[g][p][lane] = eval_program<T, SMEM, 4>(ld, sprog, spart[p], spart[p + 1] - spart[p], stk);
                }
            }
            __syncthreads();
            if (nact <= 0) continue;
            int csp = 0;  // the parts' stack is empty again: the combine reuses it
            for (int q = 0; q < nparts; q++) {
                const TreeComb c = scomb[q];
                if (q > 0) stk.set(csp++, top);
                top = partial[g][c.part][lane];
                for (int a = c.adds; a > 0; a--) top = vadd<T>(stk.get(--csp), top);
            }
        } else {
            if (nact <= 0) continue;
            top = eval_program<T, SMEM, 4>(ld, sprog, 0, sg.prog_len, stk);
        }
        char* o = out + byte;
        if (sg.rank < 0) {
            for (int d = j; d < P; d += K) st_strided<T, 32>(o + (long long)d * out_stride, top, nact);
        } else if (j == 0) {
            st_strided<T, 32>(o + (long long)sg.rank * out_stride, top, nact);
        }
    }
}

// ----------------------------------------------------------------- copies
enum CopyMode { kCopyAllgather = 0, kCopyBcast = 1, kCopyAlltoall = 2, kCopyScatter = 3, kCopyGather = 4 };

// Division of n < 2^31 by a fixed d as one multiplication and a shift
// (Granlund and Montgomery, "Division by invariant integers using
// multiplication": with l = ceil(log2 d) and m = floor(2^(31+l) / d) + 1,
// floor(n / d) = floor(n * m / 2^(31+l))).  Larger n divide directly (mul 0).
struct FastDiv {
    long long d = 1;
    unsigned mul = 0;
    int shift = 0;
    FastDiv() = default;
    FastDiv(long long divisor, long long max_n) : d(divisor) {
        if (max_n >= (1ll << 31) || divisor >= (1ll << 31)) return;
        int l = 0;
        while ((1ll << l) < divisor) l++;
        shift = 31 + l;
        mul = (unsigned)((1ull << shift) / (unsigned long long)divisor + 1);
    }
    __device__ __forceinline__ long long operator()(long long n) const {
        return mul ? (long long)(((unsigned long long)(unsigned)n * mul) >> shift) : n / d;
    }
};

// A copy collective is a set of "pairs" (source row piece, destination row
// pieces) of `unit` bytes each; unit = one rank's block.
struct CopyArgs {
    const char* in;
    long long in_stride;
    char* out;
    long long out_stride;
    int P;
    int root;
    long long unit;    // bytes per block
    int dgroups;       // k_copy_rows (allgather, bcast): destination groups per source element (>= 1)
    // k_copy_blocks, k_copy_shift: a pair is cut into `chunks` pieces.
    long long groups;  // pairs * chunks
    long long chunks;
    int tp_log2;       // k_copy_blocks: log2 of the threads per piece
    FastDiv by_chunks, by_ranks;
};

// Source of pair `i` (alltoall: block `to` of row `from`), and its
// destination in the collectives that have one.
template <int MODE>
__device__ __forceinline__ const char* copy_src(const CopyArgs& a, long long i, long long from, long long to) {
    if (MODE == kCopyAllgather) return a.in + i * a.in_stride;
    if (MODE == kCopyBcast) return a.in + (long long)a.root * a.in_stride;
    if (MODE == kCopyAlltoall) return a.in + from * a.in_stride + to * a.unit;
    if (MODE == kCopyScatter) return a.in + (long long)a.root * a.in_stride + i * a.unit;
    return a.in + i * a.in_stride;  // gather
}
template <int MODE>
__device__ __forceinline__ char* copy_dst(const CopyArgs& a, long long i, long long from, long long to) {
    if (MODE == kCopyAlltoall) return a.out + to * a.out_stride + from * a.unit;
    if (MODE == kCopyScatter) return a.out + i * a.out_stride;
    return a.out + (long long)a.root * a.out_stride + i * a.unit;  // gather
}

// The element type U of these kernels is the widest whose size divides every
// address, stride and block length of the call (uint4 when all are on the
// 16-byte grid).
//
template <typename U>
__device__ __forceinline__ void st_unit(U* p, U v) {
    if constexpr (sizeof(U) == 16) st_stream(p, v);
    else *p = v;  // partial sectors: the neighbours' parts meet in L2 (bcast, P = 8, 1,000,003 int32: 8.5 us, 12.8 with .cs)
}

// The broadcasting collectives (each element to P rows): E elements per
// thread, 32 apart, over the elements of all blocks in order.  Calls with few
// source elements split each element's destinations over `dgroups` threads
// (each loads it and stores to its share of the rows), so that small calls
// still fill the GPU.
template <int MODE, typename U, int E>
__global__ void __launch_bounds__(kThreads, 2048 / kThreads) k_copy_rows(CopyArgs a) {
    const long long nu = a.unit / (long long)sizeof(U);
    const long long step = (long long)gridDim.x * blockDim.x;
    const int G = a.dgroups;
    const long long n = (MODE == kCopyBcast ? 1 : a.P) * nu;
    const long long per = E == 1 ? n : (n + 32 * E - 1) / (32 * E) * 32, total = per * G;  // threads: whole warps
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += step) {
        const long long gi = G == 1 ? 0 : w / per, r = w - gi * per;
        const long long x0 = E == 1 ? r : (r - (r & 31)) * E + (r & 31);
        U v[E];
#pragma unroll
        for (int u = 0; u < E; u++) {
            const long long x = x0 + 32 * u;
            if (E > 1 && x >= n) continue;  // the last warp's
            const long long i = MODE == kCopyBcast ? 0 : x / nu;
            v[u] = ld_unit(reinterpret_cast<const U*>(copy_src<MODE>(a, i, 0, 0)) + (x - i * nu));
        }
        // One group: no divisions (allgather of 36 floats at P = 2: 1.95 us, 2.11 with them).
        const int d0 = G == 1 ? 0 : (int)(a.P * gi / G), d1 = G == 1 ? a.P : (int)(a.P * (gi + 1) / G);
        char* q = a.out + (long long)d0 * a.out_stride + x0 * (long long)sizeof(U);
        // Unrolled for element stores only: 16-byte stores run ahead of the
        // other blocks' (allgather, P = 128, 32 KiB: 90.1 us, 93.4 unrolled).
#pragma unroll(sizeof(U) == 16 ? 1 : 4)
        for (int d = d0; d < d1; d++, q += a.out_stride) {
            if (MODE == kCopyBcast && d == a.root) continue;
#pragma unroll
            for (int u = 0; u < E; u++)
                if (E == 1 || x0 + 32 * u < n) st_unit(reinterpret_cast<U*>(q) + 32 * u, v[u]);
        }
    }
}

// Blocks of fewer elements than k_copy_blocks takes, with one destination, and calls
// of at most kCopySmallMax: up to four elements per thread and round, over
// the elements of all blocks in order (I: the index type, 32 bits where the
// element count allows), as many threads as elements where the grid holds them.
constexpr int kCopySmallMax = 262144;
template <int MODE, typename U, typename I>
__global__ void __launch_bounds__(kThreads) k_copy_small(CopyArgs a) {
    const I nu = (I)(a.unit / (long long)sizeof(U)), P = (I)a.P;
    const long long total = (MODE == kCopyAlltoall ? (long long)a.P * a.P : a.P) * (a.unit / (long long)sizeof(U));
    const long long step = (long long)gridDim.x * blockDim.x;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += 4 * step) {
        U v[4];
        U* q[4];
#pragma unroll
        for (int x = 0; x < 4; x++) {
            if (w + x * step >= total) continue;
            const I e = (I)(w + x * step), i = e / nu, j = e - i * nu;
            const I from = MODE == kCopyAlltoall ? i / P : 0, to = i - from * P;
            v[x] = ld_unit(reinterpret_cast<const U*>(copy_src<MODE>(a, i, from, to)) + j);
            q[x] = reinterpret_cast<U*>(copy_dst<MODE>(a, i, from, to)) + j;
        }
#pragma unroll
        for (int x = 0; x < 4; x++)
            if (w + x * step < total) st_unit(q[x], v[x]);
    }
}

// Blocks of at least kCopy[Vec]BlockMin elements with one destination (alltoall,
// scatter, gather): a group of 2^tp_log2 threads moves a piece of up to E
// elements per thread, 2^tp_log2 apart, so that a warp's accesses are
// contiguous runs, E loads are in flight before the stores, and the block
// numbers are divided out once per thread instead of once per element.
// Bound by HBM.  Against one element per thread and grid step (us, B200):
// alltoall at P = 64 with 64 KiB blocks 89 -> 82, P = 256 with 516-byte blocks
// 38 -> 25.
constexpr int kCopyBlockMin = 17;     // elements of up to 8 bytes
constexpr int kCopyVecBlockMin = 16;  // 16-byte vectors
template <int MODE, typename U>
__global__ void __launch_bounds__(kThreads) k_copy_blocks(CopyArgs a) {
    constexpr int E = sizeof(U) == 16 ? 4 : 8;
    const int tp = 1 << a.tp_log2;
    const long long nu = a.unit / (long long)sizeof(U);
    const long long step = (long long)gridDim.x * blockDim.x >> a.tp_log2;
    const int t = threadIdx.x & (tp - 1);
    for (long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> a.tp_log2; w < a.groups; w += step) {
        const long long i = a.chunks == 1 ? w : a.by_chunks(w);
        const long long first = (w - i * a.chunks) * (tp * E) + t;
        const long long from = MODE == kCopyAlltoall ? a.by_ranks(i) : 0, to = i - from * a.P;
        const int have = (int)min((long long)E, (nu - first + tp - 1) >> a.tp_log2);
        const U* src = reinterpret_cast<const U*>(copy_src<MODE>(a, i, from, to)) + first;
        U* dst = reinterpret_cast<U*>(copy_dst<MODE>(a, i, from, to)) + first;
        U v[E];
#pragma unroll
        for (int u = 0; u < E; u++)
            if (u < have) v[u] = ld_unit(src + u * tp);
#pragma unroll
        for (int u = 0; u < E; u++)
            if (u < have) st_cs(dst + u * tp, v[u]);
    }
}

// Allgather and bcast off the 16-byte grid: every row receives the same
// sequence of n bytes, but the rows start at different offsets within 16
// bytes.  A block stages one tile of the sequence in shared memory once per
// such offset (16 / sizeof(U) copies, each shifted by one element more), so
// that the body of every row's tile is one bulk copy (cp.async.bulk, 16-byte
// aligned on both sides) from the copy that matches the row; the up to 30
// bytes before and after it are element stores.  Rows are split into groups
// to give the GPU about kSpreadItems blocks per SM.
//
// Bound by HBM writes (bcast at P = 96, 1,000,001 int32: 87 % of the copy
// rate): element stores off the grid leave two partial sectors per 128 bytes.
// Measured on B200 (us): bcast at P = 96,
// 1,000,001 int32 116 -> 73, allgather at P = 41, 20,001 floats 40.1 ->
// 28.5.  Rows on the grid need no staging and stay with k_copy_rows (allgather
// at P = 96, 32 KiB: 52.4 there, 58 here).
constexpr int kSpreadThreads = 128;
constexpr int kSpreadTile = 4096;  // bytes of the sequence per block
constexpr int kSpreadItems = 20;
struct SpreadArgs {
    const char* in;
    long long in_stride;
    char* out;
    long long out_stride;
    int P, skip;      // skip: the row that already holds the sequence, or -1
    long long n;      // bytes of the sequence
    long long unit;   // bytes of one contiguous source piece (n: one piece)
    int groups;       // row groups
    long long ntiles;
    FastDiv by_tiles, by_unit;  // by_unit: elements of type U
};

__device__ __forceinline__ void bulk_store(void* dst, uint32_t src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(src), "r"(bytes)
                 : "memory");
}

template <typename U>
__global__ void __launch_bounds__(kSpreadThreads) k_spread(const SpreadArgs a) {
    constexpr int kVar = 16 / sizeof(U);
    constexpr int kBatch = 8;
    __shared__ __align__(128) char sbuf[kVar][kSpreadTile];
    const long long g = a.by_tiles(blockIdx.x), x0 = (blockIdx.x - g * a.ntiles) * kSpreadTile;
    const int n = (int)min((long long)kSpreadTile, a.n - x0), nu = n / (int)sizeof(U);
    const long long u0 = x0 / (long long)sizeof(U), pu = a.unit / (long long)sizeof(U);
    for (int b = threadIdx.x; b < nu; b += kBatch * kSpreadThreads) {
        U v[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int x = b + u * kSpreadThreads;
            if (x < nu) {
                const long long e = u0 + x, i = a.unit == a.n ? 0 : a.by_unit(e);
                v[u] = ld_unit(reinterpret_cast<const U*>(a.in + i * a.in_stride) + (e - i * pu));
            }
        }
#pragma unroll
        for (int u = 0; u < kBatch; u++) {
            const int x = b + u * kSpreadThreads;
            if (x < nu) {
#pragma unroll
                for (int s = 0; s < kVar; s++)
                    if (x >= s) *reinterpret_cast<U*>(sbuf[s] + (x - s) * (int)sizeof(U)) = v[u];
            }
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the bulk copies read what this thread wrote
    __syncthreads();
    const uint32_t sb = (uint32_t)__cvta_generic_to_shared(sbuf);
    const int d0 = (int)(a.P * g / a.groups), d1 = (int)(a.P * (g + 1) / a.groups);
    for (int d = d0 + threadIdx.x; d < d1; d += kSpreadThreads) {
        if (d == a.skip) continue;
        char* dst = a.out + (long long)d * a.out_stride + x0;
        const int head = min(n, (int)(16 - ((uintptr_t)dst & 15)) & 15), body = (n - head) & ~15;
        if (body > 0) bulk_store(dst + head, sb + head / (int)sizeof(U) * kSpreadTile, body);
        for (int x = 0; x < head; x += (int)sizeof(U)) *reinterpret_cast<U*>(dst + x) = *reinterpret_cast<U*>(sbuf[0] + x);
        for (int x = head + body; x < n; x += (int)sizeof(U))
            *reinterpret_cast<U*>(dst + x) = *reinterpret_cast<U*>(sbuf[0] + x);
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // shared memory is read before the block ends
}

// Blocks whose source and destination do not share a 16-byte grid (alltoall,
// scatter, gather): 16-byte loads on the source's grid, realigned in
// registers, 16-byte stores on the destination's.  A warp copies kShiftVecs
// destination vectors of one block; a lane's vector is cut from the aligned
// source vector it loaded and the next one, which lane + 1 loaded (lane 31:
// lane 0's of the next 32).  Only source vectors that lie inside the block
// are read, so up to 31 bytes at a block's start and 47 at its end are
// copied as elements of type U.
//
// Stores are whole sectors, where element stores off the grid leave two
// partial sectors per 128 bytes.  Bound by load latency: 78 registers for
// 4-byte elements leave three blocks per SM (30 % of the warps; DRAM at 57 % of
// its peak, 78 % of the copy rate).  Measured on B200 (us, one element per
// thread -> this kernel): alltoall at P = 64 with blocks of 10,001 int32 158
// -> 64, of 10,001 bytes 153 -> 18.8; P = 128 with 2,052-byte blocks 37.4 ->
// 16.7.
constexpr int kShiftVecs = 128;  // destination vectors per warp
template <int MODE, typename U>
__global__ void __launch_bounds__(kThreads) k_copy_shift(CopyArgs a) {
    constexpr int kE = kShiftVecs / 32;
    const int lane = threadIdx.x & 31;
    const long long step = (long long)gridDim.x * (kThreads / 32);
    for (long long w = (long long)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); w < a.groups; w += step) {
        const long long i = a.chunks == 1 ? w : a.by_chunks(w);
        const long long chunk = w - i * a.chunks;
        const long long from = MODE == kCopyAlltoall ? a.by_ranks(i) : 0, to = i - from * a.P;
        const char* src = copy_src<MODE>(a, i, from, to);
        char* dst = copy_dst<MODE>(a, i, from, to);
        // Destination vectors [0, nvec) start `head` bytes into the block;
        // source vector k of its own grid starts at src + head - off + 16k,
        // and destination vector k takes bytes off.. of vectors k and k + 1.
        const int head = (int)(16 - ((uintptr_t)dst & 15)) & 15;
        const int off = (int)((uintptr_t)(src + head) & 15);
        const long long nvec = (a.unit - head) / 16;
        const long long k0 = head >= off ? 0 : 1, k1 = max(k0, min(nvec, (a.unit - head + off) / 16 - 1));
        const char* s = src + head - off;
        char* d = dst + head;
        const long long kb = chunk * (32 * kE) + lane;
        uint4 v[kE + 1];
#pragma unroll
        for (int j = 0; j <= kE; j++) {
            const long long k = kb + 32 * j;
            v[j] = make_uint4(0, 0, 0, 0);
            if (k >= k0 && k <= k1 && (j < kE || lane == 0)) v[j] = ld_stream(s + 16 * k);
        }
        uint4 t = v[0];  // the vectors one lane up, of this 32 and of the next
        auto up = [&](uint4 x) {
            const int from = (lane + 1) & 31;
            return make_uint4(__shfl_sync(0xffffffffu, x.x, from), __shfl_sync(0xffffffffu, x.y, from),
                              __shfl_sync(0xffffffffu, x.z, from), __shfl_sync(0xffffffffu, x.w, from));
        };
        t = up(v[0]);
        const int q = off >> 2, b = (off & 3) * 8;
#pragma unroll
        for (int j = 0; j < kE; j++) {
            const uint4 tn = up(v[j + 1]);
            const uint4 n = lane == 31 ? tn : t;
            t = tn;
            uint32_t x[8] = {v[j].x, v[j].y, v[j].z, v[j].w, n.x, n.y, n.z, n.w};
            if (q & 2) {
#pragma unroll
                for (int z = 0; z < 6; z++) x[z] = x[z + 2];
            }
            if (q & 1) {
#pragma unroll
                for (int z = 0; z < 5; z++) x[z] = x[z + 1];
            }
            const long long k = kb + 32 * j;
            if (k >= k0 && k < k1)
                st_stream(d + 16 * k,
                          make_uint4(__funnelshift_r(x[0], x[1], b), __funnelshift_r(x[1], x[2], b),
                                     __funnelshift_r(x[2], x[3], b), __funnelshift_r(x[3], x[4], b)));
        }
        if (chunk == 0) {
            const int n = (int)min(a.unit, head + 16 * k0) / (int)sizeof(U);
            for (int e = lane; e < n; e += 32) reinterpret_cast<U*>(dst)[e] = reinterpret_cast<const U*>(src)[e];
        }
        if (chunk == a.chunks - 1) {
            const long long from = min(a.unit, head + 16 * k1) / (long long)sizeof(U), n = a.unit / (long long)sizeof(U);
            for (long long e = from + lane; e < n; e += 32) reinterpret_cast<U*>(dst)[e] = reinterpret_cast<const U*>(src)[e];
        }
    }
}

// ------------------------------------------------------------- step engine
struct StepMove {
    int64_t dst_off, a_off, b_off;  // elements
    int32_t dst_rank, a_rank, b_rank;
    uint8_t dst_buf, a_buf, b_buf, add;
};
struct StepChunk {  // elements [start, start + n) of move `move`
    int32_t move, pad;
    int64_t start, n;
};
struct StepBufs {
    char* base[3];       // send, receive, workspace
    long long stride[3];  // bytes between rank rows
};

enum StepStatus { kStepOk = 0, kStepTimeout = 1 };

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid-wide barrier for a cooperative launch.  bar[0] counts arrivals,
// bar[1] is the generation; the last of `expected` arrivals (normally
// gridDim.x) opens it.  The wait is bounded by `timeout_ns` of %globaltimer
// and by an iteration cap; on expiry the block records kStepTimeout in
// *status and returns false (the caller then exits, so the other blocks time
// out too instead of waiting forever).
__device__ __forceinline__ bool grid_barrier(unsigned* bar, int* status, unsigned long long timeout_ns,
                                             unsigned expected) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        __threadfence();
        const unsigned gen = ld_acquire(&bar[1]);
        const unsigned arrived = atomicAdd(&bar[0], 1u);
        if (arrived == expected - 1) {
            bar[0] = 0;
            __threadfence();
            st_release(&bar[1], gen + 1);
        } else {
            const unsigned long long t0 = globaltimer_ns();
            unsigned long long iters = 0;
            while (ld_acquire(&bar[1]) == gen) {
                if (++iters > (1ull << 40) || globaltimer_ns() - t0 > timeout_ns ||
                    *(volatile int*)status != kStepOk) {
                    atomicCAS(status, kStepOk, kStepTimeout);
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

template <typename T>
__device__ __forceinline__ void run_chunk(const StepBufs& B, const StepMove& m, const StepChunk& ch) {
    constexpr long long es = sizeof(T);
    char* d = B.base[m.dst_buf] + (long long)m.dst_rank * B.stride[m.dst_buf] + (m.dst_off + ch.start) * es;
    const char* a = B.base[m.a_buf] + (long long)m.a_rank * B.stride[m.a_buf] + (m.a_off + ch.start) * es;
    const char* b = B.base[m.b_buf] + (long long)m.b_rank * B.stride[m.b_buf] + (m.b_off + ch.start) * es;
    const long long bytes = ch.n * es;
    const bool vec = (((uintptr_t)d | (uintptr_t)a | (uintptr_t)(m.add ? b : a)) & 15) == 0 && (bytes & 15) == 0;
    if (vec) {
        const long long nv = bytes / 16;
        for (long long i = threadIdx.x; i < nv; i += blockDim.x) {
            // Plain (coherent) loads: earlier levels of this launch wrote
            // these rows.
            uint4 v = ld_plain(a + i * 16);
            if (m.add) v = vadd<T>(v, ld_plain(b + i * 16));
            *(uint4*)(d + i * 16) = v;
        }
    } else {
        for (long long i = threadIdx.x; i < ch.n; i += blockDim.x) {
            T v = ((volatile const T*)a)[i];
            if (m.add) v = add_exact<T>(v, ((volatile const T*)b)[i]);
            ((T*)d)[i] = v;
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) k_steps(StepBufs B, const StepMove* __restrict__ moves,
                                                    const StepChunk* __restrict__ chunks,
                                                    const int* __restrict__ level_begin, int nlevels,
                                                    unsigned* bar, int* status, unsigned long long timeout_ns,
                                                    unsigned expected) {
    for (int l = 0; l < nlevels; l++) {
        for (int c = level_begin[l] + blockIdx.x; c < level_begin[l + 1]; c += gridDim.x) {
            const StepChunk ch = chunks[c];
            run_chunk<T>(B, moves[ch.move], ch);
        }
        if (l + 1 < nlevels && !grid_barrier(bar, status, timeout_ns, expected)) return;
    }
}

// ------------------------------------------------- pipelined step engine
// The schedule as a dataflow of items (packed segments of moves, one level
// each; built on the host by build_flow).  Blocks take items in index order
// from a global counter and run each one once the items it depends on are
// done, so a segment moves on to the next step as soon as the segments it
// reads and overwrites are ready: steps overlap, ports proceed
// independently, and no block waits for the slowest block of a level.
//
// Dependencies only point to earlier items, which were handed to running
// blocks before, so the waits always end; they are bounded nevertheless.
// State (zero-initialised once): done[item] holds the epoch of the call that
// completed it; ctl[0] is the next item, ctl[1] the blocks finished, ctl[2]
// the epoch of the last completed call, ctl[3 + l] the items of level l
// done.  The last block to finish resets the counters and advances the
// epoch, so consecutive launches need no memset.
struct FlowItem {
    int32_t pbeg, pend, dbeg, dend, level, pad;
};
constexpr int kFlowThreads = 256;                 // threads per block of k_flow
constexpr int kFlowBlocksPerSm = 1024 / kFlowThreads;  // resident blocks at 64 registers
constexpr int kFlowPieces = kFlowThreads;         // pieces per item, at most one per thread
constexpr int kFlowUnroll = 4;    // 16-byte units in flight per thread

__device__ __forceinline__ bool flow_wait(int dep, const unsigned* done, const unsigned* ctl,
                                          const int* level_items, unsigned target, unsigned extra, int* status,
                                          unsigned long long timeout_ns) {
    const bool item = dep >= 0;
    const unsigned* p = item ? &done[dep] : &ctl[3 + (-dep - 1)];
    const unsigned need = item ? target + extra : (unsigned)level_items[-dep - 1] + extra;
    if (item ? ld_acquire(p) == need : ld_acquire(p) >= need) return true;
    const unsigned long long t0 = globaltimer_ns();
    for (unsigned long long iters = 0;; iters++) {
        const unsigned v = ld_acquire(p);
        if (item ? v == need : v >= need) return true;
        if (iters > (1ull << 40) || globaltimer_ns() - t0 > timeout_ns || *(volatile int*)status != kStepOk) {
            atomicCAS(status, kStepOk, kStepTimeout);
            return false;
        }
        __nanosleep(32);
    }
}

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Completion is a release store after the block barrier (release is
// cumulative over the block's writes), read with acquire loads.
template <typename T>
__global__ void __launch_bounds__(kFlowThreads, kFlowBlocksPerSm) k_flow(StepBufs B, const StepMove* __restrict__ moves,
                                                      const StepChunk* __restrict__ pieces,
                                                      const FlowItem* __restrict__ items, int nitems,
                                                      const int* __restrict__ deps,
                                                      const int* __restrict__ level_items, int nlevels,
                                                      unsigned* done, unsigned* ctl, int* status,
                                                      unsigned long long timeout_ns, unsigned extra) {
    __shared__ long long s_pref[kFlowPieces + 1];  // first unit of each piece
    __shared__ char* s_d[kFlowPieces];
    __shared__ const char* s_a[kFlowPieces];
    __shared__ const char* s_b[kFlowPieces];
    __shared__ long long s_nvec[kFlowPieces];      // 16-byte units of the body
    __shared__ unsigned char s_head[kFlowPieces];  // element units before the body
    __shared__ unsigned char s_add[kFlowPieces];
    __shared__ long long s_warp[kFlowThreads / 32];
    __shared__ int s_item, s_ok;
    __shared__ unsigned s_target;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        const unsigned t = ld_acquire(&ctl[2]) + 1u;
        s_target = t == 0 ? 1u : t;  // 0 is the initial value of done[]
    }
    __syncthreads();
    const unsigned target = s_target;
    constexpr long long es = sizeof(T);
    for (;;) {
        if (tid == 0) s_item = *(volatile int*)status == kStepOk ? (int)atomicAdd(&ctl[0], 1u) : nitems;
        __syncthreads();
        const int i = s_item;
        if (i >= nitems) break;
        const FlowItem it = items[i];
        // Piece table (addresses; element head, 16-byte body and element
        // tail; tables only, no data rows) and a block scan of the unit
        // counts, both before the dependency wait, so that they are off the
        // critical path.  A piece whose destination and sources sit at the same
        // offset within 16 bytes gets a vector body; any other piece is
        // all element units.
        const int np = it.pend - it.pbeg;
        long long units = 0;
        if (tid < np) {
            const StepChunk ch = pieces[it.pbeg + tid];
            const StepMove m = moves[ch.move];
            char* d = B.base[m.dst_buf] + (long long)m.dst_rank * B.stride[m.dst_buf] + (m.dst_off + ch.start) * es;
            const char* a = B.base[m.a_buf] + (long long)m.a_rank * B.stride[m.a_buf] + (m.a_off + ch.start) * es;
            const char* b = B.base[m.b_buf] + (long long)m.b_rank * B.stride[m.b_buf] + (m.b_off + ch.start) * es;
            const uintptr_t mis = ((uintptr_t)d ^ (uintptr_t)a) | (m.add ? ((uintptr_t)d ^ (uintptr_t)b) : 0);
            const long long n = ch.n;
            long long head = n, nvec = 0;
            if ((mis & 15) == 0) {
                head = min((long long)((16 - ((uintptr_t)d & 15)) & 15) / es, n);
                nvec = (n - head) * es / 16;
            }
            units = n - nvec * (16 / es) + nvec;
            s_d[tid] = d;
            s_a[tid] = a;
            s_b[tid] = b;
            s_nvec[tid] = nvec;
            s_head[tid] = (unsigned char)min(head, 255ll);
            s_add[tid] = m.add ? 1 : 0;
        }
        long long inc = units;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) s_warp[warp] = inc;
        __syncthreads();
        long long before = 0;
        for (int w = 0; w < warp; w++) before += s_warp[w];
        s_pref[tid + 1] = before + inc;
        if (tid == 0) s_pref[0] = 0;
        // The dependency wait comes last, so that only one block barrier
        // separates the last dependency's completion from this item's loads.
        if (warp == 0) {
            bool ok = true;
            for (int d = it.dbeg + lane; d < it.dend && ok; d += 32)
                ok = flow_wait(deps[d], done, ctl, level_items, target, extra, status, timeout_ns);
            ok = __all_sync(0xffffffffu, ok);
            if (lane == 0) s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) break;  // a wait expired; the status is recorded
        const long long total = s_pref[np];
        int cur = 0;
        for (long long u0 = tid; u0 < total; u0 += (long long)kFlowUnroll * kFlowThreads) {
            uint4 va[kFlowUnroll], vb[kFlowUnroll];  // a vector, or an element in the low bytes
            char* dp[kFlowUnroll];
            int kind[kFlowUnroll];  // -1: none; bit 0: add, bit 1: vector
#pragma unroll
            for (int k = 0; k < kFlowUnroll; k++) {
                const long long u = u0 + (long long)k * kFlowThreads;
                kind[k] = -1;
                if (u < total) {
                    if (!(u >= s_pref[cur] && u < s_pref[cur + 1])) {
                        int lo = 0, hi = np - 1;  // last piece starting at or before u
                        while (lo < hi) {
                            const int mid = (lo + hi + 1) >> 1;
                            if (s_pref[mid] <= u) lo = mid; else hi = mid - 1;
                        }
                        cur = lo;
                    }
                    const long long r = u - s_pref[cur];
                    const long long head = s_head[cur], nvec = s_nvec[cur];
                    const int add = s_add[cur];
                    // Plain (coherent) loads: other blocks wrote these rows
                    // during this launch.
                    if (r >= head && r < head + nvec) {
                        const long long off = head * es + (r - head) * 16;
                        kind[k] = add | 2;
                        dp[k] = s_d[cur] + off;
                        va[k] = ld_plain(s_a[cur] + off);
                        if (add) vb[k] = ld_plain(s_b[cur] + off);
                    } else {
                        const long long e = r < head ? r : r - nvec + nvec * (16 / es);
                        kind[k] = add;
                        dp[k] = s_d[cur] + e * es;
                        *(T*)&va[k] = *((volatile const T*)s_a[cur] + e);
                        if (add) *(T*)&vb[k] = *((volatile const T*)s_b[cur] + e);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kFlowUnroll; k++) {
                if (kind[k] < 0) continue;
                if (kind[k] & 2)
                    *(uint4*)dp[k] = (kind[k] & 1) ? vadd<T>(va[k], vb[k]) : va[k];
                else
                    *(T*)dp[k] = (kind[k] & 1) ? add_exact<T>(*(const T*)&va[k], *(const T*)&vb[k]) : *(const T*)&va[k];
            }
        }
        __syncthreads();
        if (tid == 0) {
            st_release(&done[i], target);
            red_release_add(&ctl[3 + it.level], 1u);
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&ctl[1], 1u) == gridDim.x - 1) {
            ctl[0] = 0;
            ctl[1] = 0;
            for (int l = 0; l < nlevels; l++) ctl[3 + l] = 0;
            __threadfence();
            st_release(&ctl[2], target);
        }
    }
}

// ------------------------------------------- pipelined engine, fused passes
// The same dataflow driver as k_flow over a fused schedule (level fusion,
// bine_plan.h): a piece belongs to a fused move whose value is a postfix
// program over at most kFuseLeaves state elements, written to at most
// kFuseDsts destinations.  Each unit (a 16-byte vector, or an element at a
// piece's unaligned head and tail) loads its leaves eight at a time,
// evaluates the program in the order of the original levels' additions (full
// binary trees in registers, others on a five-entry stack in shared memory),
// and stores the value to every destination; all loads come before the
// stores, so a move may update its own elements in place.  Items of copies
// only (the gather and alltoall passes) move four 16-byte units per thread
// and round, other items one unit with eight leaves in flight.  The planner
// cuts each pass into a whole multiple of the resident blocks' count of
// equal-traffic items.
//
// Bound by DRAM and L2 traffic for large rows, by the chain of dependent loads
// per item (three table rounds, the wait, the data) for small ones.  Programs
// of up to 16 leaves instead of 8 take allreduce B at P = 256 from 1.34 to
// 1.13 times the algorithmic bytes and from four passes to three; us per call
// on B200, float32, 8 leaves -> 16: 1 MiB per rank 165 -> 129, 4 MiB 564 ->
// 442, 400,004 bytes 154 -> 105; P = 96, 4 MiB 305 -> 202; P = 64, 8 KiB 20.5
// -> 16.9; reduce_scatter at P = 128, 1 MiB 62 -> 44.  Schedules of copies
// have a form of their own (FusedItemSmem<1>: 14 of 47 KiB, 64 registers,
// four blocks per SM instead of three of 80): alltoall at P = 128, 1 MiB 128
// -> 107 us; in the 16-leaf form it took 142.
struct FusedMoveDev {
    int64_t n;
    int32_t leaf_begin, nleaves, dst_begin, ndst;
};
struct FusedLeafDev {
    int32_t rank;
    uint8_t buf, adds, pad[2];
    int64_t off;
};
struct FusedDstDev {
    int32_t rank;
    uint8_t buf, pad[3];
    int64_t off;
};
constexpr int kFuseLeaves = 16;
constexpr int kFuseDsts = 8;
constexpr int kFuseDepth = 5;      // evaluation stack, the top included
constexpr int kFuseRound = 8;      // leaves of a 16-byte unit loaded at once
constexpr int kFusedPieces = 128;  // pieces per item, at most one per thread
static_assert(kFusedPieces <= kFlowThreads, "one thread per piece of an item");

// Per-item tables of k_flow_fused: every piece's leaf and destination
// addresses, its evaluation program, and block scans of its 16-byte units
// and of its element units (an unaligned head and tail, or the whole piece
// when its rows are not mutually 16-byte aligned).  The planner keeps an
// item below 2^31 elements, so unit counts fit 32 bits.
template <int L>
struct FusedItemSmem {
    int pref[kFusedPieces + 1];   // first 16-byte unit of each piece
    int epref[kFusedPieces + 1];  // first element unit of each piece
    const char* leaf[kFusedPieces][L];
    char* dst[kFusedPieces][kFuseDsts];
    long long start[kFusedPieces], n[kFusedPieces];
    int nvec[kFusedPieces], lb[kFusedPieces], db[kFusedPieces];
    unsigned char adds[kFusedPieces][L];
    unsigned char head[kFusedPieces], nl[kFusedPieces], nd[kFusedPieces];
    unsigned char full[kFusedPieces];  // the program is a full binary tree
    uint4 stk[L > 1 ? kFuseDepth - 1 : 1][L > 1 ? kFlowThreads : 1];  // evaluation stack below the top, per thread
    char* base[3];               // the launch's buffer rows (StepBufs), read from shared memory
    long long stride[3];
    long long warp_sum[kFlowThreads / 32];
    int item, ok, maxnl;
    unsigned target;
};

// Last piece of the item whose units (prefix table pref) start at or
// before unit u; cur is the guess.
__device__ __forceinline__ int fused_piece(const int* pref, int u, int np, int cur) {
    if (u >= pref[cur] && u < pref[cur + 1]) return cur;
    int lo = 0, hi = np - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (pref[mid] <= u) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// The 16-byte units of an item of copies: U units per thread and round, every
// unit's load issued before the round's stores.  Units of one item touch
// disjoint elements apart from a move's in-place reads of its own elements,
// so the order of rounds and units does not matter.
template <typename T, int U, int L>
__device__ __forceinline__ void fused_units_copy(const FusedItemSmem<L>& S, int tid, int total, int np) {
    constexpr int es = sizeof(T);
    int cur = 0;
    for (int u0 = tid; u0 < total; u0 += U * kFlowThreads) {
        uint4 v[U];
        int pc[U], off[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
            const int u = u0 + k * kFlowThreads;
            pc[k] = -1;
            off[k] = 0;
            if (u < total) {
                cur = fused_piece(S.pref, u, np, cur);
                pc[k] = cur;
                off[k] = S.head[cur] * es + (u - S.pref[cur]) * 16;
                v[k] = ld_plain(S.leaf[cur][0] + off[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
            if (pc[k] < 0) continue;
            const int p = pc[k];
            const int nd = S.nd[p];
#pragma unroll
            for (int j = 0; j < kFuseDsts; j++)
                if (j < nd) *(uint4*)(S.dst[p][j] + off[k]) = v[k];
        }
    }
}

// The value of one unit of piece p (V: a 16-byte vector, or one element),
// leaves loaded eight at a time by ld(leaf).  Full binary trees (the sums of
// the halving and butterfly steps) are added in registers; other programs
// keep the entries below the top of their stack in this thread's column of
// S.stk (registers would cost the third block per SM).  IEEE and wrapping
// integer addition are commutative, so only the tree's shape matters, and it
// is the program's.
template <typename V, int L, typename Ld, typename Add>
__device__ __forceinline__ V fused_value(FusedItemSmem<L>& S, int tid, int p, Ld ld, Add add) {
    static_assert(kFuseRound == 8 && L == 16, "two rounds of eight leaves");
    const int nl = S.nl[p];
    V v[kFuseRound];
    if (S.full[p]) {  // 1, 2, 4, 8 or 16 leaves
#pragma unroll
        for (int j = 0; j < kFuseRound; j++)
            if (j < nl) v[j] = ld(S.leaf[p][j]);
        V top = v[0];
        if (nl > 1) top = add(top, v[1]);
        if (nl > 2) top = add(top, add(v[2], v[3]));
        if (nl > 4) top = add(top, add(add(v[4], v[5]), add(v[6], v[7])));
        if (nl > 8) {
#pragma unroll
            for (int j = 0; j < kFuseRound; j++) v[j] = ld(S.leaf[p][kFuseRound + j]);
            top = add(top, add(add(add(v[0], v[1]), add(v[2], v[3])), add(add(v[4], v[5]), add(v[6], v[7]))));
        }
        return top;
    }
    V top;
    int sp = 0;
#pragma unroll 1
    for (int r = 0; r < nl; r += kFuseRound) {
#pragma unroll
        for (int j = 0; j < kFuseRound; j++)
            if (r + j < nl) v[j] = ld(S.leaf[p][r + j]);
#pragma unroll
        for (int j = 0; j < kFuseRound; j++)
            if (r + j < nl) {
                if (r + j > 0) *(V*)&S.stk[sp++][tid] = top;
                top = v[j];
                for (int a = S.adds[p][r + j]; a > 0; a--) top = add(*(const V*)&S.stk[--sp][tid], top);
            }
    }
    return top;
}

// The 16-byte units of any item, one per thread and round.
template <typename T, int L>
__device__ __forceinline__ void fused_units_wide(FusedItemSmem<L>& S, int tid, int total, int np) {
    constexpr int es = sizeof(T);
    int cur = 0;
    for (int u = tid; u < total; u += kFlowThreads) {
        cur = fused_piece(S.pref, u, np, cur);
        const int off = S.head[cur] * es + (u - S.pref[cur]) * 16, nd = S.nd[cur];
        const uint4 val = fused_value<uint4>(S, tid, cur, [&](const char* p) { return ld_plain(p + off); },
                                             [](uint4 x, uint4 y) { return vadd<T>(x, y); });
#pragma unroll
        for (int j = 0; j < kFuseDsts; j++)
            if (j < nd) *(uint4*)(S.dst[cur][j] + off) = val;
    }
}

// The element units of an item: a piece's unaligned head, its tail after
// the 16-byte body, or all of a piece without one.
template <typename T, int L>
__device__ __forceinline__ void fused_elements(FusedItemSmem<L>& S, int tid, int total, int np) {
    constexpr int per_vec = 16 / sizeof(T);
    int cur = 0;
    for (int u = tid; u < total; u += kFlowThreads) {
        cur = fused_piece(S.epref, u, np, cur);
        const long long r = u - S.epref[cur];
        const long long e = r < S.head[cur] ? r : r + (long long)S.nvec[cur] * per_vec;
        const int nd = S.nd[cur];
        T val;
        if constexpr (L == 1)
            val = *((volatile const T*)S.leaf[cur][0] + e);
        else
            val = fused_value<T>(S, tid, cur, [&](const char* p) { return *((volatile const T*)p + e); },
                                 [](T x, T y) { return add_exact<T>(x, y); });
#pragma unroll
        for (int j = 0; j < kFuseDsts; j++)
            if (j < nd) *((T*)S.dst[cur][j] + e) = val;
    }
}

// L: the longest program of the schedule, 1 (copies only) or kFuseLeaves.
template <typename T, int L>
__global__ void __launch_bounds__(kFlowThreads, L == 1 ? 4 : 3) k_flow_fused(StepBufs B, const FusedMoveDev* __restrict__ moves,
                                                            const FusedLeafDev* __restrict__ leaves,
                                                            const FusedDstDev* __restrict__ dsts,
                                                            const StepChunk* __restrict__ pieces,
                                                            const FlowItem* __restrict__ items, int nitems,
                                                            const int* __restrict__ deps,
                                                            const int* __restrict__ level_items, int nlevels,
                                                            unsigned* done, unsigned* ctl, int* status,
                                                            unsigned long long timeout_ns, unsigned extra) {
    __shared__ FusedItemSmem<L> S;
    static_assert(sizeof(FusedItemSmem<L>) <= 48 * 1024, "static shared memory");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        const unsigned t = ld_acquire(&ctl[2]) + 1u;
        S.target = t == 0 ? 1u : t;
    }
    if (tid < 3) {
        S.base[tid] = B.base[tid];
        S.stride[tid] = B.stride[tid];
    }
    __syncthreads();
    const unsigned target = S.target;
    constexpr long long es = sizeof(T);
    constexpr int kSlots = L + kFuseDsts;
    for (;;) {
        if (tid == 0) {
            S.item = *(volatile int*)status == kStepOk ? (int)atomicAdd(&ctl[0], 1u) : nitems;
            S.maxnl = 1;
        }
        __syncthreads();
        const int i = S.item;
        if (i >= nitems) break;
        const FlowItem it = items[i];
        const int np = it.pend - it.pbeg;  // at most kFusedPieces (the planner's bound)
        // The item's tables in three rounds of independent loads, all before
        // the dependency wait: pieces and moves, then every leaf and
        // destination address, then each piece's vector body and units.
        if (tid < np) {
            const StepChunk ch = pieces[it.pbeg + tid];
            const FusedMoveDev m = moves[ch.move];
            S.start[tid] = ch.start;
            S.n[tid] = ch.n;
            S.lb[tid] = m.leaf_begin;
            S.db[tid] = m.dst_begin;
            S.nl[tid] = (unsigned char)m.nleaves;
            S.nd[tid] = (unsigned char)m.ndst;
            atomicMax(&S.maxnl, m.nleaves);
        }
        __syncthreads();
#pragma unroll 4
        for (int e = tid; e < np * kSlots; e += kFlowThreads) {
            const int p = e / kSlots, j = e % kSlots;
            if (j < L) {
                if (j < S.nl[p]) {
                    const FusedLeafDev lf = leaves[S.lb[p] + j];
                    S.leaf[p][j] =
                        S.base[lf.buf] + (long long)lf.rank * S.stride[lf.buf] + (lf.off + S.start[p]) * es;
                    S.adds[p][j] = lf.adds;
                }
            } else if (j - L < S.nd[p]) {
                const FusedDstDev d = dsts[S.db[p] + j - L];
                S.dst[p][j - L] =
                    S.base[d.buf] + (long long)d.rank * S.stride[d.buf] + (d.off + S.start[p]) * es;
            }
        }
        __syncthreads();
        // Both unit counts in one scan: element units in the high half.
        long long units = 0;
        if (tid < np) {
            const uintptr_t first = (uintptr_t)S.leaf[tid][0];
            uintptr_t mis = 0;
            for (int j = 1; j < S.nl[tid]; j++) mis |= (uintptr_t)S.leaf[tid][j] ^ first;
            for (int j = 0; j < S.nd[tid]; j++) mis |= (uintptr_t)S.dst[tid][j] ^ first;
            const long long n = S.n[tid];
            long long head = 0, nvec = 0;
            if ((mis & 15) == 0) {
                head = min((long long)((16 - (first & 15)) & 15) / es, n);
                nvec = (n - head) * es / 16;
            }
            units = ((n - nvec * (16 / es)) << 32) | nvec;
            S.nvec[tid] = (int)nvec;
            S.head[tid] = (unsigned char)head;
            const int nl = S.nl[tid];
            bool full = (nl & (nl - 1)) == 0;
            for (int j = 1; j < nl; j++) full = full && S.adds[tid][j] == __ffs(j + 1) - 1;
            S.full[tid] = full;
        }
        long long inc = units;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += v;
        }
        if (lane == 31) S.warp_sum[warp] = inc;
        __syncthreads();
        long long before = 0;
        for (int w = 0; w < warp; w++) before += S.warp_sum[w];
        if (tid < kFusedPieces) {
            S.pref[tid + 1] = (int)((before + inc) & 0xffffffffll);
            S.epref[tid + 1] = (int)((before + inc) >> 32);
        }
        if (tid == 0) S.pref[0] = S.epref[0] = 0;
        if (warp == 0) {
            bool ok = true;
            for (int d = it.dbeg + lane; d < it.dend && ok; d += 32)
                ok = flow_wait(deps[d], done, ctl, level_items, target, extra, status, timeout_ns);
            ok = __all_sync(0xffffffffu, ok);
            if (lane == 0) S.ok = ok;
        }
        __syncthreads();
        if (!S.ok) break;  // a wait expired; the status is recorded
        const int total = S.pref[np];
        if (L == 1 || S.maxnl <= 1)
            fused_units_copy<T, 4>(S, tid, total, np);
        else if constexpr (L > 1)
            fused_units_wide<T>(S, tid, total, np);
        if (S.epref[np] > 0) fused_elements<T>(S, tid, S.epref[np], np);
        __syncthreads();
        if (tid == 0) {
            st_release(&done[i], target);
            red_release_add(&ctl[3 + it.level], 1u);
        }
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&ctl[1], 1u) == gridDim.x - 1) {
            ctl[0] = 0;
            ctl[1] = 0;
            for (int l = 0; l < nlevels; l++) ctl[3 + l] = 0;
            __threadfence();
            st_release(&ctl[2], target);
        }
    }
}

}  // namespace dev
}  // namespace bine

// ------------------------------------------------------ torus link bytes
// Per-link byte accounting of a schedule on the communicator's torus.  A
// message takes the dimension-ordered route, minimal on each ring, the +
// direction on ties (Bine and recursive-doubling peers differ in one
// coordinate; 1-D algorithms on a torus may differ in several).  Link (node, d, dir) has index (node*ndims + d)*2 + dir
// (dir 0: +, 1: -).  Each message adds its bytes to a cyclic range of link
// positions on one ring, recorded as two or three signed updates of a
// difference array (unsigned wrap-around arithmetic, exact mod 2^64); one
// prefix scan per ring then yields the counts.  Cost: O(messages + links)
// instead of O(messages * hops).
#include "bine_sched.h"

namespace bine {
namespace dev {

__device__ __forceinline__ size_t link_index(const Torus& t, int node, int d, int dir) {
    return ((size_t)node * t.ndims + d) * 2 + dir;
}

// Adds `bytes` to the links of the route src -> dst: dimension-ordered
// (dimension 0 first), minimal in each dimension, + direction on ties.
__device__ __forceinline__ void add_route(const Torus& t, int src, int dst, unsigned long long bytes,
                                          unsigned long long* diff) {
    if (src == dst || bytes == 0) return;
    int a[kMaxDims] = {0, 0, 0}, b[kMaxDims] = {0, 0, 0};
    t.coords(src, a);
    t.coords(dst, b);
    int c[kMaxDims] = {a[0], a[1], a[2]};
    const unsigned long long neg = 0ull - bytes;
    for (int d = 0; d < t.ndims; d++) {
        if (c[d] == b[d]) continue;
        const int L = t.dims[d];
        const int delta = pmod(b[d] - c[d], L);
        int dir = 0, start = c[d], hops = delta;
        if (L - delta < delta) {  // minus direction: positions c-h+1 .. c
            dir = 1;
            hops = L - delta;
            start = pmod(c[d] - hops + 1, L);
        }
        auto at = [&](int pos) {
            int q[kMaxDims] = {c[0], c[1], c[2]};
            q[d] = pos;
            return link_index(t, t.id(q), d, dir);
        };
        const int end = start + hops;  // exclusive
        atomicAdd(&diff[at(start)], bytes);
        if (end < L) {
            atomicAdd(&diff[at(end)], neg);
        } else if (end > L) {  // wraps: [start, L) and [0, end - L)
            atomicAdd(&diff[at(0)], bytes);
            atomicAdd(&diff[at(end - L)], neg);
        }
        c[d] = b[d];
    }
}

// One thread per message (src, dst, elements) of a host-planned schedule.
__global__ void k_link_from_msgs(Torus t, const long long* __restrict__ msgs, long long n, int es,
                                 unsigned long long* diff) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        add_route(t, (int)msgs[4 * i + 1], (int)msgs[4 * i + 2], (unsigned long long)msgs[4 * i + 3] * es, diff);
}

struct LinkGen {
    Torus t;
    int family, ports, kind;  // kind 0: bandwidth-optimal allreduce, 1: latency-optimal allreduce,
                              //      2: contiguous allgather (distance halving)
    long long count;          // the collective's count argument
    int es;
};

// One thread per (rank, port): generates the messages of the schedule
// directly from the step math (power-of-two torus dimensions only, where
// every binomial tree visits each rank once).
//   kind 0: the reduce-scatter message of rank r at step i carries the
//   blocks of the subtree reached through peer_i(r) with later steps (the
//   blocks whose block_step is i); the allgather sends the same volume back.
//   kind 1: the full port slice to peer_i(r) at every step.
//   kind 2: 2^s blocks to peer_{S-1-s}(r) at step s.
__global__ void k_link_generate(LinkGen g, unsigned long long* diff) {
    const long long total = (long long)g.t.size * g.ports;
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < total; w += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(w / g.ports), port = (int)(w % g.ports);
        StepDim sd[kMaxSteps];
        step_dims(g.t, port, sd);
        const int S = g.t.num_steps, P = g.t.size;
        const long long cp = g.count / g.ports + (port < g.count % g.ports ? 1 : 0);
        if (g.kind == 1) {
            for (int i = 0; i < S; i++)
                add_route(g.t, r, step_peer_rank(g.t, sd, i, port, g.family, r), (unsigned long long)cp * g.es, diff);
            continue;
        }
        if (g.kind == 2) {
            // Allgather blocks: by block, then port (count per block = count).
            const long long b0 = g.count / g.ports + (port < g.count % g.ports ? 1 : 0);
            for (int s = 0; s < S; s++)
                add_route(g.t, r, step_peer_rank(g.t, sd, S - 1 - s, port, g.family, r),
                          ((unsigned long long)1 << s) * b0 * g.es, diff);
            continue;
        }
        const long long q = cp / P, rem = cp % P;
        for (int i = 0; i < S; i++) {
            const int child = step_peer_rank(g.t, sd, i, port, g.family, r);
            // Iterative walk of child's subtree along steps > i.
            int stk_node[kMaxSteps * (kMaxSteps + 1) / 2 + 1];
            int8_t stk_step[kMaxSteps * (kMaxSteps + 1) / 2 + 1];
            int sp = 0;
            stk_node[sp] = child;
            stk_step[sp++] = (int8_t)(i + 1);
            unsigned long long elems = 0;
            while (sp > 0) {
                const int node = stk_node[--sp];
                const int st = stk_step[sp];
                elems += (unsigned long long)(q + (node < rem ? 1 : 0));
                for (int j = st; j < S; j++) {
                    stk_node[sp] = step_peer_rank(g.t, sd, j, port, g.family, node);
                    stk_step[sp++] = (int8_t)(j + 1);
                }
            }
            add_route(g.t, r, child, elems * g.es, diff);  // reduce-scatter step i
            add_route(g.t, child, r, elems * g.es, diff);  // allgather step S-1-i
        }
    }
}

// The same schedules ring by ring, for tori whose rings hold at most
// kLinkMaxRing nodes: one block per ring (a torus line of dimension d), in
// one launch that writes every link once.
//
// Every message of these schedules moves along one dimension, so a ring's
// link loads depend only on the messages between its own nodes.  At step k
// of dimension d node p exchanges with q = peer_k(p) and q with p (the step
// is an involution), so the difference entries at p come from p's own
// message and the one it receives: each thread adds both to its own
// entries, with no atomics, and a block scan turns them into loads.
//
// Message sizes of kind 0 need, per node, the number of ranks below `rem`
// (the blocks one element longer) in the subtree it reaches with the steps
// after k.  That subtree is a product over the dimensions of one-dimensional
// subtrees (a step of one dimension leaves the other coordinates alone), and
// "below rem" is lexicographic in the coordinates, so
//
//   f = sum over dims e of prod_{e' < e} M_e' * G_e * prod_{e' > e} Z_e'
//
// with G_e the members of dimension e's subtree below rem's coordinate, M_e
// those equal to it and Z_e its size.  G and M obey G_k(c) = G_{k+1}(c) +
// G_{k+1}(peer_k(c)), one addition per node and step, in place in shared
// memory.
//
// k_link_generate walks each subtree node by node instead (P nodes per rank,
// a serial chain on a local stack) and adds with global atomics, after a
// memset and before k_link_scan.  It took 4,788 us of device time on the
// 64x64 torus (allreduce B, 1 port) and the scan 48 us, 4,827 us per call;
// with this kernel a call takes 16.4 us, bound by the latency of its steps
// (a barrier pair and some hundred instructions each, 18 of them there).
// The walk remains for rings beyond kLinkMaxRing, whose tables do not fit
// in shared memory (24 bytes per node).
constexpr int kLinkMaxRing = 8192;

// Peer of coordinate c at a step of signed distance `dist` (Bine; negated
// for odd coordinates) or of XOR distance `dist` (recursive doubling).
__device__ __forceinline__ int ring_peer(bool xored, int dist, int L, int c) {
    return xored ? c ^ dist : (c + ((c & 1) ? -dist : dist)) & (L - 1);
}

__global__ void __launch_bounds__(1024) k_link_rings(LinkGen g, int maxring, unsigned long long* __restrict__ links) {
    extern __shared__ unsigned long long ring_smem[];
    unsigned long long* dplus = ring_smem;        // + direction: difference entry of position p
    unsigned long long* dminus = dplus + maxring;  // - direction: difference entry of position p + 1
    int* cnt = (int*)(dminus + maxring);           // G of the current dimension at the current step
    int* mem = cnt + maxring;                      // M
    __shared__ StepDim sd[kMaxSteps];
    __shared__ int8_t after[kMaxSteps][kMaxDims];  // steps of each dimension among steps 0..i
    __shared__ int8_t at[kMaxDims][kMaxSteps];     // global step of (dimension, step)
    __shared__ int dist[kMaxSteps];                // of a ring's step k on the current port
    __shared__ int tabg[kMaxDims][kMaxSteps + 1], tabm[kMaxDims][kMaxSteps + 1];
    __shared__ unsigned long long wsum[4][32];
    const Torus& t = g.t;
    const int S = t.num_steps, tid = threadIdx.x, nth = blockDim.x;
    // The ring: dimension d, the other coordinates in c.
    int line = blockIdx.x, d = 0;
    while (d + 1 < t.ndims && line >= t.size / t.dims[d]) line -= t.size / t.dims[d++];
    int c[kMaxDims] = {0, 0, 0};
    for (int i = t.ndims - 1; i >= 0; i--) {
        if (i == d) continue;
        c[i] = line % t.dims[i];
        line /= t.dims[i];
    }
    const int L = t.dims[d], Lm = L - 1;  // every dimension is a power of two here
    const bool xored = g.family == kFamilyRecDoub;
    for (int p = tid; p < L; p += nth) dplus[p] = dminus[p] = 0;
    unsigned long long wp = 0, wm = 0;  // bytes of this thread's ranges that pass position 0
    for (int port = 0; port < g.ports; port++) {
        const long long cp = g.count / g.ports + (port < g.count % g.ports ? 1 : 0);
        const long long q0 = cp >> S;  // 2^S ranks
        const int rem = (int)(cp & (t.size - 1));
        const bool uneven = g.kind == 0 && rem > 0;
        int R[kMaxDims] = {0, 0, 0};
        t.coords(rem, R);
        __syncthreads();  // the previous port's tables are consumed
        if (tid >= 32 - kMaxSteps && tid < 32) {
            const int k = tid - (32 - kMaxSteps);
            dist[k] = xored ? 1 << k : (mirrored_port(port, t.ndims) ? -rho(k) : rho(k));
        }
        if (tid == 0) {
            step_dims(t, port, sd);
            int8_t n[kMaxDims] = {0, 0, 0};
            for (int i = 0; i < S; i++) {
                at[sd[i].d][sd[i].k] = (int8_t)i;
                n[sd[i].d]++;
                for (int e = 0; e < kMaxDims; e++) after[i][e] = n[e];
            }
        }
        // One dimension's G and M after every step, last step first: the
        // other dimensions' at this ring's coordinates go to the tables.
        auto begin = [&](int e) {
            for (int p = tid; p < t.dims[e]; p += nth) {
                cnt[p] = p < R[e];
                mem[p] = p == R[e];
            }
            __syncthreads();
        };
        auto advance = [&](int e, int k) {
            for (int p = tid; p < t.dims[e]; p += nth) {
                const int q = ring_peer(xored, dist[k], t.dims[e], p);
                if (p < q) {
                    cnt[p] = cnt[q] = cnt[p] + cnt[q];
                    mem[p] = mem[q] = mem[p] + mem[q];
                }
            }
            __syncthreads();
        };
        if (uneven) {
            for (int e = 0; e < t.ndims; e++) {
                if (e == d) continue;
                begin(e);
                for (int k = t.steps_per_dim[e]; k >= 0; k--) {
                    if (tid == 0) {
                        tabg[e][k] = cnt[c[e]];
                        tabm[e][k] = mem[c[e]];
                    }
                    if (k > 0) {
                        __syncthreads();
                        advance(e, k - 1);
                    }
                }
                __syncthreads();  // cnt and mem are reused for the next dimension
            }
            begin(d);
        } else {
            __syncthreads();
        }
        for (int k = t.steps_per_dim[d] - 1; k >= 0; k--) {
            const int i = at[d][k];
            // f(x) = alpha * G(x) + beta * M(x) + gamma at this step.
            long long alpha = 0, beta = 0, gamma = 0;
            if (uneven) {
                long long pre = 1, pre_d = 1;  // products of M: all dims before e; without dimension d
                for (int e = 0; e < t.ndims; e++) {
                    long long post = 1;
                    for (int h = e + 1; h < t.ndims; h++) post <<= t.steps_per_dim[h] - after[i][h];
                    if (e == d) {
                        alpha = pre * post;
                    } else {
                        const int ke = after[i][e];
                        if (e < d) gamma += pre * tabg[e][ke] * post;
                        else beta += pre_d * tabg[e][ke] * post;
                        if (e < d) pre *= tabm[e][ke];
                        pre_d *= tabm[e][ke];
                    }
                }
            }
            for (int p = tid; p < L; p += nth) {
                const int q = ring_peer(xored, dist[k], L, p);
                unsigned long long bytes;
                if (g.kind == 1) {
                    bytes = (unsigned long long)cp;
                } else if (g.kind == 2) {
                    bytes = (unsigned long long)cp << (S - 1 - i);
                } else {  // the reduce-scatter message one way and the allgather's from the peer
                    bytes = 2ull * ((unsigned long long)q0 << (S - 1 - i));
                    if (uneven) bytes += alpha * (cnt[p] + cnt[q]) + beta * (mem[p] + mem[q]) + 2 * gamma;
                }
                bytes *= g.es;
                // p's message to q takes the shorter way round (+ on ties),
                // and so does q's to p.
                const int h = (q - p) & Lm;
                unsigned long long dp = 0, dm = 0;
                if (h + h <= L) {  // + : positions p .. p + h - 1
                    dp += bytes;
                    if (p + h >= L) wp += bytes;
                } else {  // - : positions q + 1 .. p
                    dm -= bytes;
                    if (((q + 1) & Lm) + (L - h) >= L) wm += bytes;
                }
                if (h + h >= L) dp -= bytes;  // q's message comes in the + direction and ends before p
                else dm += bytes;             // or in the - direction, from position p + 1 on
                dplus[p] += dp;
                dminus[p] += dm;
            }
            if (uneven && k > 0) {
                __syncthreads();
                advance(d, k);
            }
        }
    }
    __syncthreads();
    // Scan: thread tid owns positions [tid * per, +per).
    const int per = (L + nth - 1) / nth, p0 = min(L, tid * per), p1 = min(L, p0 + per);
    unsigned long long sp = 0, sm = 0;
    for (int p = p0; p < p1; p++) {
        sp += dplus[p];
        sm += dminus[p];
    }
    const int lane = tid & 31, warp = tid >> 5;
    unsigned long long ip = sp, im = sm;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long a = __shfl_up_sync(0xffffffffu, ip, o), b = __shfl_up_sync(0xffffffffu, im, o);
        if (lane >= o) {
            ip += a;
            im += b;
        }
        wp += __shfl_xor_sync(0xffffffffu, wp, o);
        wm += __shfl_xor_sync(0xffffffffu, wm, o);
    }
    if (lane == 31) {
        wsum[0][warp] = ip;
        wsum[1][warp] = im;
        wsum[2][warp] = wp;
        wsum[3][warp] = wm;
    }
    __syncthreads();
    unsigned long long ap = ip - sp, am = im - sm;  // exclusive prefixes
    unsigned long long tp = 0, tm = dminus[L - 1];
    for (int w = 0; w < nth / 32; w++) {
        if (w < warp) {
            ap += wsum[0][w];
            am += wsum[1][w];
        }
        tp += wsum[2][w];
        tm += wsum[3][w];
    }
    size_t li = link_index(t, t.id(c), d, 0);  // c[d] = 0: position 0
    size_t step = 2 * t.ndims;                 // links of consecutive positions
    for (int e = d + 1; e < t.ndims; e++) step *= t.dims[e];
    for (int p = p0; p < p1; p++) {
        ap += dplus[p];
        links[li + p * step] = tp + ap;      // prefix including position p
        links[li + p * step + 1] = tm + am;  // entries of positions 0..p, each one place to the left
        am += dminus[p];
    }
}

// One thread per ring: prefix sums of the difference array, in place.
__global__ void k_link_scan(Torus t, unsigned long long* links) {
    long long nlines = 0;
    long long base[kMaxDims];
    for (int d = 0; d < t.ndims; d++) {
        base[d] = nlines;
        nlines += 2ll * (t.size / t.dims[d]);
    }
    for (long long w = (long long)blockIdx.x * blockDim.x + threadIdx.x; w < nlines; w += (long long)gridDim.x * blockDim.x) {
        int d = 0;
        while (d + 1 < t.ndims && w >= base[d + 1]) d++;
        const long long k = w - base[d];
        const int dir = (int)(k & 1);
        long long line = k >> 1;  // index over the other coordinates
        int c[kMaxDims] = {0, 0, 0};
        for (int i = t.ndims - 1; i >= 0; i--) {
            if (i == d) continue;
            c[i] = (int)(line % t.dims[i]);
            line /= t.dims[i];
        }
        unsigned long long acc = 0;
        for (int p = 0; p < t.dims[d]; p++) {
            c[d] = p;
            const size_t li = link_index(t, t.id(c), d, dir);
            acc += links[li];
            links[li] = acc;
        }
    }
}

}  // namespace dev
}  // namespace bine

// --------------------------------------------------------- batched launch
// Thousands of independent allreduce / reduce_scatter / allgather calls of
// different P, sizes and element types in ONE launch.  Every call is cut
// into tiles; blocks take tiles grid-stride from the global tile range and
// find their call by a binary search over tile_begin, bounded by a table of
// the calls at every kBatchHint-th tile (no table up to kBatchHint tiles,
// where it holds one range: a small call with its data outside L2 takes 6.1
// us, 8.2 with the table's dependent load; both forms in one kernel cost
// batches of 100 calls 2 us).  Reduction tiles are `tc` 16-byte
// columns wide and split the P rows over 256/tc row groups (tc comes from
// the tuning: narrow tiles with many row groups for large P, wide tiles for
// small P); allgather tiles are 256 vectors of the flattened (source rank,
// column) space, each stored to at most kBatchRows rows, so that a tile
// writes about as much as a reduction tile moves: with all P rows in one
// tile a few tiles of 2 MB ended a small batch (64 calls, 55 MB: 49 us).
// Integer sums wrap, float32 sums accumulate in FP64 (the FAST order).
//
// Bound by HBM.  B200, us per launch with the default tuning, against tiles of
// all rows, a search of all calls and a grid of the resident blocks: 512 mixed
// calls of up to 64 KiB (1.97 GB) 386 -> 332, 400 of up to 500 bytes on up to
// 512 ranks 98.8 -> 61.6, 60 of those 39.0 -> 16.4.
namespace bine {
namespace dev {

enum BatchOp { kBatchAllreduce = 0, kBatchReduceScatter = 1, kBatchAllgather = 2 };

struct BatchItem {
    const char* in;
    char* out;
    long long in_stride, out_stride;  // bytes between rank rows
    long long ncol;                   // 16-byte vectors per input row
    long long blk;                    // reduce_scatter: vectors per destination rank
    long long tile_begin, ntiles;
    int P, op, is_float, tc;
    int rgroups;                      // allgather: row groups; tile = group * vector tiles + vector tile
    int pad;
};
constexpr int kBatchRows = 32;
constexpr int kBatchHint = 64;

template <typename T, typename A>
__device__ __forceinline__ void batch_reduce_tile(const BatchItem& it, long long tile, Lanes<float, double>* part_f,
                                                  uint4* res) {
    const int tc = it.tc, groups = kThreads / tc;
    const int lane = threadIdx.x % tc, grp = threadIdx.x / tc;
    const int per = (it.P + groups - 1) / groups;
    const int r0 = min(it.P, grp * per), r1 = min(it.P, r0 + per);
    const long long col = tile * tc + lane;
    Lanes<T, A> acc;
    acc.zero();
    if (col < it.ncol) {
        const char* p = it.in + col * 16;
        int r = r0;
        for (; r + 8 <= r1; r += 8) {
            uint4 v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = ld_stream(p + (long long)(r + u) * it.in_stride);
#pragma unroll
            for (int u = 0; u < 8; u++) acc.add(v[u]);
        }
        for (; r < r1; r++) acc.add(ld_stream(p + (long long)r * it.in_stride));
    }
    Lanes<T, A>* part = reinterpret_cast<Lanes<T, A>*>(part_f);
    part[threadIdx.x] = acc;
    __syncthreads();
    if (grp == 0) {
        Lanes<T, A> s = part[lane];
        for (int g = 1; g < groups; g++)
#pragma unroll
            for (int i = 0; i < Lanes<T, A>::N; i++) s.v[i] = add_exact<A>(s.v[i], part[g * tc + lane].v[i]);
        res[lane] = s.pack();
    }
    __syncthreads();
    if (col < it.ncol) {
        const uint4 v = res[lane];
        if (it.op == kBatchAllreduce) {
            char* q = it.out + col * 16;
            for (int d = grp; d < it.P; d += groups) st_stream(q + (long long)d * it.out_stride, v);
        } else if (grp == 0) {
            const long long owner = col / it.blk;
            st_stream(it.out + owner * it.out_stride + (col - owner * it.blk) * 16, v);
        }
    }
}

// Four blocks per SM: 64 registers keep a reduction tile's eight loads in
// flight.  With the 46 to 48 that the compiler takes unasked, float tiles of
// many rows wait for them in turn (us, 48 registers / 64: one call of 888 floats
// on 456 ranks 14.4 / 10.9, of 40 floats on 521 ranks outside L2 26.6 / 14.5).
template <bool TABLE>
__global__ void __launch_bounds__(kThreads, 4) k_batch(const BatchItem* __restrict__ items, int nitems,
                                                    const int* __restrict__ hint, long long total_tiles) {
    __shared__ Lanes<float, double> part[kThreads];
    __shared__ uint4 res[kThreads];
    for (long long t = blockIdx.x; t < total_tiles; t += gridDim.x) {
        int lo = TABLE ? hint[t / kBatchHint] : 0, hi = TABLE ? hint[t / kBatchHint + 1] : nitems - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (items[mid].tile_begin <= t) lo = mid;
            else hi = mid - 1;
        }
        const BatchItem it = items[lo];
        const long long tile = t - it.tile_begin;
        if (it.op == kBatchAllgather) {
            const int vtiles = (int)(it.ntiles / it.rgroups), g = (int)(tile / vtiles);
            const long long idx = (tile - (long long)g * vtiles) * kThreads + threadIdx.x;
            if (idx < (long long)it.P * it.ncol) {
                const long long i = idx / it.ncol, j = idx - i * it.ncol;
                const uint4 v = ld_stream(it.in + i * it.in_stride + j * 16);
                const int d0 = (int)((long long)it.P * g / it.rgroups), d1 = (int)((long long)it.P * (g + 1) / it.rgroups);
                char* q = it.out + (long long)d0 * it.out_stride + idx * 16;
                for (int d = d0; d < d1; d++, q += it.out_stride) st_stream(q, v);
            }
        } else if (it.is_float) {
            batch_reduce_tile<float, double>(it, tile, part, res);
        } else {
            batch_reduce_tile<int32_t, int32_t>(it, tile, part, res);
        }
        __syncthreads();
    }
}

}  // namespace dev
}  // namespace bine
