// Device kernels shared by the setup and the solve: block-sparse products, block
// Jacobi, transfers, chunked reductions. See solver.cuh for the data layout.
#pragma once
#include "solver.cuh"

namespace sc {

// y = A x;  y += A x;  y = r - A x;  y = x + step D^-1 (r - A x);  y = A x and y2 = step D^-1 y (step
// null: 1)
enum SpmvMode { SPMV_Y = 0, SPMV_ADD = 1, SPMV_RES = 2, SPMV_RES_SMOOTH = 3, SPMV_Y_JACOBI = 4 };

__device__ __forceinline__ int64_t lower_bound_i32(const int32_t* __restrict__ a, int64_t lo, int64_t hi, int32_t v) {
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (a[mid] < v)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

template <class T>
__device__ __forceinline__ void ld6(const T* __restrict__ p, T (&o)[6]) {
    if constexpr (sizeof(T) == 8) {
        const double2* q = reinterpret_cast<const double2*>(p);
        double2 a = q[0], b = q[1], c = q[2];
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y; o[4] = c.x; o[5] = c.y;
    } else {
        const float2* q = reinterpret_cast<const float2*>(p);
        float2 a = q[0], b = q[1], c = q[2];
        o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y; o[4] = c.x; o[5] = c.y;
    }
}
template <class T>
__device__ __forceinline__ void st6(T* __restrict__ p, const T (&o)[6]) {
    if constexpr (sizeof(T) == 8) {
        double2* q = reinterpret_cast<double2*>(p);
        q[0] = make_double2(o[0], o[1]);
        q[1] = make_double2(o[2], o[3]);
        q[2] = make_double2(o[4], o[5]);
    } else {
        float2* q = reinterpret_cast<float2*>(p);
        q[0] = make_float2(o[0], o[1]);
        q[1] = make_float2(o[2], o[3]);
        q[2] = make_float2(o[4], o[5]);
    }
}

// ---- reductions over a level's chunks ----------------------------------------------------
// A sum over a piece is taken in one fixed order whatever the launch: a chunk (CHUNK parts)
// has 256 lanes, lane t adds the chunk's values t, t + 256, ... in turn; the lanes' sums meet
// in a halving tree (t + 128, + 64, ..., + 1); 32 strided lanes add the piece's chunks and
// meet in a tree again.
//
// The order leaves each lane a serial chain of up to 96 values, and the launch decides where
// the lanes run. WHOLE: a block a chunk, a thread a lane. SPLIT, where that would leave most
// of the device idle: a block 32 lanes of a chunk, whose eight warps bring the lanes' values
// to shared memory (a warp alone gets one load in some 55 cycles) and whose first warp runs
// the chains from there. The last of a chunk's blocks to arrive adds its lanes, the last of
// a piece's chunks the piece, so no launch follows for the sums or for the scalars that
// come of them.
constexpr int RED_LANES = 256;
struct Chunks {
    const int64_t* lo = nullptr;           // nchunks + 1 bounds, in parts
    const int32_t* piece = nullptr;        // each chunk's piece
    const int64_t* piece_chunk = nullptr;  // each piece's first chunk
    double* part = nullptr;                // two partial sums a chunk
    double* lanes = nullptr;               // SPLIT: two sums a lane of a chunk
    uint32_t* arrived = nullptr;           // SPLIT: per chunk, warps that arrived (zero between kernels)
    uint32_t* ticket = nullptr;            // per piece, chunks that arrived (zero between kernels)
};
// A block a chunk fills the device from about four blocks an SM on (148 of them; where the
// line lies changes no sum's order).
constexpr int64_t RED_WHOLE = 592;
inline bool red_split(int64_t nchunks) { return nchunks < RED_WHOLE; }
inline unsigned red_grid(int64_t nchunks) { return (unsigned)(red_split(nchunks) ? 8 * nchunks : nchunks); }
constexpr int RED_STEPS = 6 * CHUNK / RED_LANES;  // a lane's values at most
template <bool SPLIT>
constexpr size_t red_smem(int streams) { return SPLIT ? (size_t)streams * RED_STEPS * 32 * sizeof(double) : 0; }

// This thread's chunk and lane.
template <bool SPLIT>
__device__ __forceinline__ int red_chunk() {
    return SPLIT ? (int)(blockIdx.x >> 3) : (int)blockIdx.x;
}
template <bool SPLIT>
__device__ __forceinline__ int red_lane() {
    return SPLIT ? (int)((blockIdx.x & 7) * 32 + (threadIdx.x & 31)) : (int)threadIdx.x;
}

// A lane's chain: use(i, load(i)) for i = first, first + 256, ... below end, in that order, U
// loads in flight.
template <int U, class F, class G>
__device__ __forceinline__ void red_chain(int64_t first, int64_t end, F&& load, G&& use) {
    using V = decltype(load(first));
    int64_t i = first;
    for (; i + RED_LANES * (U - 1) < end; i += RED_LANES * U) {
        V v[U];
#pragma unroll
        for (int j = 0; j < U; j++) v[j] = load(i + RED_LANES * j);
#pragma unroll
        for (int j = 0; j < U; j++) use(i + RED_LANES * j, v[j]);
    }
    V v[U];
#pragma unroll
    for (int j = 0; j < U; j++)
        if (i + RED_LANES * j < end) v[j] = load(i + RED_LANES * j);
#pragma unroll
    for (int j = 0; j < U; j++)
        if (i + RED_LANES * j < end) use(i + RED_LANES * j, v[j]);
}

// This lane's values from first to end, S numbers each, in order. WHOLE: load(i, v), then
// use(v), U values' loads in flight. SPLIT: the block's warps load, and its first warp uses;
// false in the others, whose part ends here. sm: red_smem(S) bytes.
template <bool SPLIT, int S, int U, class F, class G>
__device__ __forceinline__ bool red_run(double* sm, int64_t first, int64_t end, F&& load, G&& use) {
    if constexpr (!SPLIT) {
        struct V {
            double v[S];
        };
        red_chain<U>(
            first, end,
            [&](int64_t i) {
                V x;
                load(i, x.v);
                return x;
            },
            [&](int64_t, const V& x) { use(x.v); });
        return true;
    } else {
        const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
        constexpr int PER = RED_STEPS / 8;  // a warp's steps: w, w + 8, ...
        double v[PER][S];
#pragma unroll
        for (int u = 0; u < PER; u++)
            if (first + RED_LANES * (int64_t)(w + 8 * u) < end) load(first + RED_LANES * (int64_t)(w + 8 * u), v[u]);
#pragma unroll
        for (int u = 0; u < PER; u++)
            if (first + RED_LANES * (int64_t)(w + 8 * u) < end)
#pragma unroll
                for (int q = 0; q < S; q++) sm[(q * RED_STEPS + w + 8 * u) * 32 + l] = v[u][q];
        __syncthreads();
        if (w != 0) return false;
        const int n = first < end ? (int)((end - first + RED_LANES - 1) / RED_LANES) : 0;
#pragma unroll 8
        for (int k = 0; k < n; k++) {
            double x[S];
#pragma unroll
            for (int q = 0; q < S; q++) x[q] = sm[(q * RED_STEPS + k) * 32 + l];
            use(x);
        }
        return true;
    }
}

// Every thread that red_run left going comes here with its lane's sums a and b. True in one thread of
// the last warp to arrive of the chunk's piece, with the piece's sums in a and b.
template <bool SPLIT>
__device__ __forceinline__ bool red_finish(const Chunks& ch, int c, int t, int p, double& a, double& b) {
    double va[8], vb[8];
    const int l = threadIdx.x & 31;
    if constexpr (SPLIT) {
        double* ln = ch.lanes + 2 * RED_LANES * (int64_t)c;
        __stcg(ln + t, a);
        __stcg(ln + RED_LANES + t, b);
        __threadfence();
        __syncwarp();
        uint32_t n = 0;
        if (l == 0) n = atomicAdd(ch.arrived + c, 1u);
        if (__shfl_sync(0xffffffffu, n, 0) != 7) return false;
        if (l == 0) ch.arrived[c] = 0;
        __threadfence();
#pragma unroll
        for (int k = 0; k < 8; k++) {
            va[k] = __ldcg(ln + l + 32 * k);
            vb[k] = __ldcg(ln + RED_LANES + l + 32 * k);
        }
    } else {
        __shared__ double ra[RED_LANES], rb[RED_LANES];
        ra[t] = a;
        rb[t] = b;
        __syncthreads();
        if (t >= 32) return false;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            va[k] = ra[l + 32 * k];
            vb[k] = rb[l + 32 * k];
        }
    }
#pragma unroll
    for (int w = 4; w > 0; w >>= 1)
#pragma unroll
        for (int k = 0; k < w; k++) {
            va[k] += va[k + w];
            vb[k] += vb[k + w];
        }
    a = va[0];
    b = vb[0];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, off);
        b += __shfl_down_sync(0xffffffffu, b, off);
    }
    const int64_t c0 = ch.piece_chunk[p], c1 = ch.piece_chunk[p + 1];
    uint32_t n = 0;
    if (l == 0) {
        __stcg(ch.part + 2 * (int64_t)c, a);
        __stcg(ch.part + 2 * (int64_t)c + 1, b);
        __threadfence();
        n = atomicAdd(ch.ticket + p, 1u);
    }
    if (__shfl_sync(0xffffffffu, n, 0) != (uint32_t)(c1 - c0 - 1)) return false;
    if (l == 0) ch.ticket[p] = 0;
    __threadfence();
    a = b = 0.0;
#pragma unroll 8
    for (int64_t i = c0 + l; i < c1; i += 32) {
        const double2 v = __ldcg(reinterpret_cast<const double2*>(ch.part) + i);
        a += v.x;
        b += v.y;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
    }
    return l == 0;
}

// Host launchers (kernels.cu).
Chunks red_chunks(Context& ctx, const Level& L);
// nnz (the stored blocks) picks the warps a row (one when 0); see warps_per_row.
template <class T>
void spmv(Context& ctx, int mode, int64_t nrows, const int64_t* rowptr, const int32_t* col, const T* val, const T* x,
          const T* r, T* y, const T* inv, const double* step, const int32_t* piece, const int32_t* skip_row,
          const int32_t* done, int64_t nnz = 0, T* y2 = nullptr);
template <class T>
void jacobi(Context& ctx, int64_t n, const T* inv, const T* r, T* x, const double* step, const int32_t* piece,
            const int32_t* skip_row, const int32_t* done);
template <class T>
void top_solve(Context& ctx, const Level& L, const T* r, T* z, const int32_t* done);
// out[p] = sum over piece p's parts of a.b (6 values a part), deterministic.
template <class T>
void seg_dot_t(Context& ctx, const Level& L, const T* a, const T* b, double* out);

// x = A' b, A dense (n x n, row-major)
void dense_apply(Context& ctx, int64_t n, const double* A, const double* b, double* x);
// per piece the smoother's step from the last power iteration, w = D^-1 K v
void power_step(Context& ctx, const Level& L, const double* w, const double* v, double* step);

}  // namespace sc
