// Block-sparse products, block Jacobi, restriction, direct top solves and chunked
// reductions, in FP64 and FP32. All are HBM-bound streaming kernels.
#include "kernels.cuh"

namespace sc {

namespace {

// One warp per block row. Lane = 8*g + r: block slot g (4 blocks in flight per warp),
// block row r (lanes with r >= 6 idle). Each lane reads one 6-value row of a block
// (48 B FP64 / 24 B FP32, contiguous across the 6 lanes of a slot) and the 6 values of
// x at the block's column.
template <class T, int MODE>
__global__ void __launch_bounds__(256) k_spmv(int64_t nrows, const int64_t* __restrict__ rowptr,
                                              const int32_t* __restrict__ col, const T* __restrict__ val,
                                              const T* __restrict__ x, const T* __restrict__ r, T* __restrict__ y,
                                              const T* __restrict__ inv, const double* __restrict__ step,
                                              const int32_t* __restrict__ piece, const int32_t* __restrict__ skip_row,
                                              const int32_t* __restrict__ done, T* __restrict__ y2) {
    int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (row >= nrows) return;
    int lane = threadIdx.x & 31;
    // the loads that wait for nothing, before the checks that wait for some of them
    int64_t e0 = rowptr[row], e1 = rowptr[row + 1];
    const int32_t skip = skip_row ? skip_row[row] : 0;
    int p = piece ? piece[row] : 0;
    if (skip || (done && done[p])) return;
    int g = lane >> 3, rr = lane & 7;
    T acc = T(0);
    if (rr < 6) {
        // two of the slot's blocks (e, e + 4) loaded before either is used: 8 blocks in
        // flight per warp; the lane still adds its blocks in the order e0 + g, + 4, + 8, ...
        int64_t e = e0 + g;
        for (; e + 4 < e1; e += 8) {
            int32_t j0 = col[e], j1 = col[e + 4];
            T a0[6], x0[6], a1[6], x1[6];
            ld6<T>(val + 36 * e + 6 * rr, a0);
            ld6<T>(val + 36 * (e + 4) + 6 * rr, a1);
            ld6<T>(x + 6 * (int64_t)j0, x0);
            ld6<T>(x + 6 * (int64_t)j1, x1);
#pragma unroll
            for (int c = 0; c < 6; c++) acc = fma(a0[c], x0[c], acc);
#pragma unroll
            for (int c = 0; c < 6; c++) acc = fma(a1[c], x1[c], acc);
        }
        if (e < e1) {
            int32_t j = col[e];
            T a[6], xv[6];
            ld6<T>(val + 36 * e + 6 * rr, a);
            ld6<T>(x + 6 * (int64_t)j, xv);
#pragma unroll
            for (int c = 0; c < 6; c++) acc = fma(a[c], xv[c], acc);
        }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    // lanes 0..5 hold row values
    if (MODE == SPMV_Y) {
        if (lane < 6) y[6 * row + lane] = acc;
    } else if (MODE == SPMV_ADD) {
        if (lane < 6) y[6 * row + lane] += acc;
    } else if (MODE == SPMV_RES) {
        if (lane < 6) y[6 * row + lane] = r[6 * row + lane] - acc;
    } else {
        T left = lane >= 6 ? T(0) : MODE == SPMV_Y_JACOBI ? acc : r[6 * row + lane] - acc;
        T l6[6];
#pragma unroll
        for (int c = 0; c < 6; c++) l6[c] = __shfl_sync(0xffffffffu, left, c);
        if (lane < 6) {
            const T* d = inv + 36 * row + 6 * lane;
            T s = T(0);
#pragma unroll
            for (int c = 0; c < 6; c++) s = fma(d[c], l6[c], s);
            if (MODE == SPMV_Y_JACOBI) {
                y[6 * row + lane] = acc;
                y2[6 * row + lane] = s * (step ? (T)step[p] : T(1));
            } else {
                y[6 * row + lane] = x[6 * row + lane] + (T)step[p] * s;
            }
        }
    }
}

// A row's blocks by asynchronous copies: the sum of this lane's products over its slot's
// blocks first + g, + stride, ... below e1 (lane = 8 g + r: slot g of 4, block row r, lanes
// with r >= 6 idle), a warp's groups of four consecutive blocks `stride` apart.
//
// On levels of few, long rows the product is bound by its chain row bounds -> columns -> x
// and by how many blocks a warp has in flight, eight with loads to registers. cp.async
// brings blocks and x to the warp's own ring of shared memory instead, 32 blocks ahead, 16
// bytes a lane, and the lanes add from there, in the same order: FP64 rows over four warps
// (a 32^3 piece's levels 2 and 3) 10.5-12.9 us to 7.2-9.6, over two (a 128^3 piece's level 3)
// 124-131 to 112-115. Where rows are many it only costs occupancy (a warp a row took 216 us for
// 161 in FP32, 396 for 308 in FP64), and in FP32, whose blocks are half the bytes, it gains
// nothing over two or four warps (74 us for 66, and a whole 61 x 45 x 37 solve 1 % slower):
// those keep the loads to registers (as deep a pipeline in registers was slower still).
constexpr int RING = 4, RING_BLOCKS = 8;  // stages of eight blocks: two of each slot
template <class T>
struct Ring {
    T val[RING][RING_BLOCKS * 36];
    T x[RING][RING_BLOCKS * 6];
};
__device__ __forceinline__ void cp16(void* s, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(s)), "l"(g)
                 : "memory");
}
template <class T>
__device__ __forceinline__ T row_stream(Ring<T>& ring, int64_t first, int64_t e1, int stride,
                                        const int32_t* __restrict__ col, const T* __restrict__ val,
                                        const T* __restrict__ x) {
    static_assert(sizeof(T) == 8, "the 16-byte copies of x need 16-byte parts");
    constexpr int PIECES = 36 * (int)sizeof(T) / 16;  // 16-byte pieces of a block
    const int lane = threadIdx.x & 31, g = lane >> 3, rr = lane & 7;
    T acc = T(0);
    // the columns of a turn of the ring: lane l's block is the l-th of the warp's
    auto block = [&](int64_t base, int l) { return base + (int64_t)stride * (l >> 2) + (l & 3); };
    int32_t cols = block(first, lane) < e1 ? col[block(first, lane)] : 0;
    auto issue = [&](int64_t base, int s) {  // stage s of the turn that starts at base
        const int64_t b0 = base + 2 * (int64_t)stride * s;
        for (int q = lane; q < RING_BLOCKS * PIECES; q += 32) {
            const int64_t e = block(b0, q / PIECES);
            if (e < e1)
                cp16(reinterpret_cast<char*>(ring.val[s]) + 16 * q,
                     reinterpret_cast<const char*>(val + 36 * e) + 16 * (q % PIECES));
        }
        const int32_t j = __shfl_sync(0xffffffffu, cols, 8 * s + min(lane / 3, 7));
        if (lane < 24 && block(b0, lane / 3) < e1) {
            cp16(ring.x[s] + 2 * lane, x + 6 * (int64_t)j + 2 * (lane % 3));
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
#pragma unroll
    for (int s = 0; s < RING; s++) issue(first, s);
    for (int64_t base = first; base < e1; base += 8 * (int64_t)stride) {
        const int64_t next = base + 8 * (int64_t)stride;
        if (next < e1) cols = block(next, lane) < e1 ? col[block(next, lane)] : 0;
#pragma unroll
        for (int s = 0; s < RING; s++) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(RING - 1) : "memory");
            __syncwarp();
            const int64_t b0 = base + 2 * (int64_t)stride * s + g;
            if (rr < 6) {
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (b0 + (int64_t)stride * u < e1) {
                        T a[6], xv[6];
                        ld6<T>(ring.val[s] + 36 * (4 * u + g) + 6 * rr, a);
                        ld6<T>(ring.x[s] + 6 * (4 * u + g), xv);
#pragma unroll
                        for (int c = 0; c < 6; c++) acc = fma(a[c], xv[c], acc);
                    }
            }
            __syncwarp();
            if (next < e1)
                issue(next, s);
            else
                asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    return acc;
}

// The same with each row split over WPR warps, for levels of few, long rows (coarse
// levels and their transfers), where one warp a row leaves the device idle. Warp w of a
// row takes its blocks e0 + 4 w + g, then every 4 WPR, streamed where that measured faster
// (above; the rings of more than four warps would not fit), else two in flight; the warps'
// partial sums meet in shared memory and are added in warp order (a fixed order).
template <class T, int WPR>
constexpr bool split_streams() { return sizeof(T) == 8 && (WPR == 2 || WPR == 4); }
template <class T, int WPR>
constexpr int split_warps() { return split_streams<T, WPR>() ? 4 : WPR > 8 ? WPR : 8; }
template <class T, int MODE, int WPR>
__global__ void __launch_bounds__(32 * split_warps<T, WPR>()) k_spmv_split(
    int64_t nrows, const int64_t* __restrict__ rowptr, const int32_t* __restrict__ col, const T* __restrict__ val,
    const T* __restrict__ x, const T* __restrict__ r, T* __restrict__ y, const T* __restrict__ inv,
    const double* __restrict__ step, const int32_t* __restrict__ piece, const int32_t* __restrict__ skip_row,
    const int32_t* __restrict__ done, T* __restrict__ y2) {
    constexpr int RPC = split_warps<T, WPR>() / WPR;  // rows per thread block
    constexpr int STRIDE = 4 * WPR;
    __shared__ T part[RPC * WPR][6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wr = warp % WPR;
    const int64_t row = (int64_t)blockIdx.x * RPC + warp / WPR;
    bool active = row < nrows;
    int64_t e0 = 0, e1 = 0;
    int32_t skip = 0, p = 0;
    if (active) {  // the loads that wait for nothing, before the checks that wait for some of them
        e0 = rowptr[row], e1 = rowptr[row + 1];
        if (skip_row) skip = skip_row[row];
        if (piece) p = piece[row];
        active = !(skip || (done && done[p]));
    }
    T acc = T(0);
    if constexpr (split_streams<T, WPR>()) {
        __shared__ __align__(16) Ring<T> ring[4];
        if (active) acc = row_stream<T>(ring[warp], e0 + 4 * wr, e1, 4 * WPR, col, val, x);
    } else {
        const int g = lane >> 3, rr = lane & 7;
        if (active && rr < 6) {
            int64_t e = e0 + 4 * wr + g;
            for (; e + STRIDE < e1; e += 2 * STRIDE) {
                int32_t j0 = col[e], j1 = col[e + STRIDE];
                T a0[6], x0[6], a1[6], x1[6];
                ld6<T>(val + 36 * e + 6 * rr, a0);
                ld6<T>(val + 36 * (e + STRIDE) + 6 * rr, a1);
                ld6<T>(x + 6 * (int64_t)j0, x0);
                ld6<T>(x + 6 * (int64_t)j1, x1);
#pragma unroll
                for (int c = 0; c < 6; c++) acc = fma(a0[c], x0[c], acc);
#pragma unroll
                for (int c = 0; c < 6; c++) acc = fma(a1[c], x1[c], acc);
            }
            if (e < e1) {
                int32_t j = col[e];
                T a[6], xv[6];
                ld6<T>(val + 36 * e + 6 * rr, a);
                ld6<T>(x + 6 * (int64_t)j, xv);
#pragma unroll
                for (int c = 0; c < 6; c++) acc = fma(a[c], xv[c], acc);
            }
        }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    if (lane < 6) part[warp][lane] = acc;
    __syncthreads();
    if (!active || wr != 0) return;  // whole warps
    acc = T(0);
    if (lane < 6)
#pragma unroll
        for (int w = 0; w < WPR; w++) acc += part[warp + w][lane];
    if (MODE == SPMV_Y) {
        if (lane < 6) y[6 * row + lane] = acc;
    } else if (MODE == SPMV_ADD) {
        if (lane < 6) y[6 * row + lane] += acc;
    } else if (MODE == SPMV_RES) {
        if (lane < 6) y[6 * row + lane] = r[6 * row + lane] - acc;
    } else {
        T left = lane >= 6 ? T(0) : MODE == SPMV_Y_JACOBI ? acc : r[6 * row + lane] - acc;
        T l6[6];
#pragma unroll
        for (int c = 0; c < 6; c++) l6[c] = __shfl_sync(0xffffffffu, left, c);
        if (lane < 6) {
            const T* d = inv + 36 * row + 6 * lane;
            T s = T(0);
#pragma unroll
            for (int c = 0; c < 6; c++) s = fma(d[c], l6[c], s);
            if (MODE == SPMV_Y_JACOBI) {
                y[6 * row + lane] = acc;
                y2[6 * row + lane] = s * (step ? (T)step[p] : T(1));
            } else {
                y[6 * row + lane] = x[6 * row + lane] + (T)step[p] * s;
            }
        }
    }
}

// The same with half a warp a row (two rows a warp), for rows of a few blocks (the
// level-1 prolongation: P has about nine blocks a row): lanes 8 g + r of a half, g = 0, 1,
// take the row's blocks e0 + g, then every two, two in flight.
template <class T, int MODE>
__global__ void __launch_bounds__(256) k_spmv_half(int64_t nrows, const int64_t* __restrict__ rowptr,
                                                   const int32_t* __restrict__ col, const T* __restrict__ val,
                                                   const T* __restrict__ x, const T* __restrict__ r, T* __restrict__ y,
                                                   const T* __restrict__ inv, const double* __restrict__ step,
                                                   const int32_t* __restrict__ piece,
                                                   const int32_t* __restrict__ skip_row,
                                                   const int32_t* __restrict__ done, T* __restrict__ y2) {
    const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 4;
    const int lane = threadIdx.x & 31, h = lane & 16, hl = lane & 15;
    bool active = row < nrows;
    int64_t e0 = 0, e1 = 0;
    int32_t skip = 0, p = 0;
    if (active) {
        e0 = rowptr[row], e1 = rowptr[row + 1];
        if (skip_row) skip = skip_row[row];
        if (piece) p = piece[row];
        active = !(skip || (done && done[p]));
    }
    const int g = hl >> 3, rr = hl & 7;
    T acc = T(0);
    if (active && rr < 6) {
        int64_t e = e0 + g;
        for (; e + 2 < e1; e += 4) {
            int32_t j0 = col[e], j1 = col[e + 2];
            T a0[6], x0[6], a1[6], x1[6];
            ld6<T>(val + 36 * e + 6 * rr, a0);
            ld6<T>(val + 36 * (e + 2) + 6 * rr, a1);
            ld6<T>(x + 6 * (int64_t)j0, x0);
            ld6<T>(x + 6 * (int64_t)j1, x1);
#pragma unroll
            for (int c = 0; c < 6; c++) acc = fma(a0[c], x0[c], acc);
#pragma unroll
            for (int c = 0; c < 6; c++) acc = fma(a1[c], x1[c], acc);
        }
        if (e < e1) {
            int32_t j = col[e];
            T a[6], xv[6];
            ld6<T>(val + 36 * e + 6 * rr, a);
            ld6<T>(x + 6 * (int64_t)j, xv);
#pragma unroll
            for (int c = 0; c < 6; c++) acc = fma(a[c], xv[c], acc);
        }
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    // lanes h + 0..5 hold the half's row values
    if (MODE == SPMV_Y) {
        if (active && hl < 6) y[6 * row + hl] = acc;
    } else if (MODE == SPMV_ADD) {
        if (active && hl < 6) y[6 * row + hl] += acc;
    } else if (MODE == SPMV_RES) {
        if (active && hl < 6) y[6 * row + hl] = r[6 * row + hl] - acc;
    } else {
        T left = !(active && hl < 6) ? T(0) : MODE == SPMV_Y_JACOBI ? acc : r[6 * row + hl] - acc;
        T l6[6];
#pragma unroll
        for (int c = 0; c < 6; c++) l6[c] = __shfl_sync(0xffffffffu, left, h + c);
        if (active && hl < 6) {
            const T* d = inv + 36 * row + 6 * hl;
            T s = T(0);
#pragma unroll
            for (int c = 0; c < 6; c++) s = fma(d[c], l6[c], s);
            if (MODE == SPMV_Y_JACOBI) {
                y[6 * row + hl] = acc;
                y2[6 * row + hl] = s * (step ? (T)step[p] : T(1));
            } else {
                y[6 * row + hl] = x[6 * row + hl] + (T)step[p] * s;
            }
        }
    }
}

template <class T>
__global__ void k_jacobi(int64_t n, const T* __restrict__ inv, const T* __restrict__ r, T* __restrict__ x,
                         const double* __restrict__ step, const int32_t* __restrict__ piece,
                         const int32_t* __restrict__ skip_row, const int32_t* __restrict__ done) {
    int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    T rv[6], o[6];
    ld6<T>(r + 6 * k, rv);
    const int32_t skip = skip_row ? skip_row[k] : 0;
    int p = piece ? piece[k] : 0;
    if (skip || (done && done[p])) return;
    T st = step ? (T)step[p] : T(1);
    const T* d = inv + 36 * k;
#pragma unroll
    for (int i = 0; i < 6; i++) {
        T s = T(0);
#pragma unroll
        for (int c = 0; c < 6; c++) s = fma(d[6 * i + c], rv[c], s);
        o[i] = s * st;
    }
    st6<T>(x + 6 * k, o);
}

// z_i = sum over j of A[j][i] r_j in the order of j, FP64, for the 32 rows i from i0 on. What
// bounds it is that chain and the loads it waits for (a warp alone gets one load in some 55
// cycles), so 32 rows are a block whose eight warps bring TOP_TILE values of j to shared
// memory at a time and whose first warp runs the chain: a 96-row top 30 to 4.6 us, a
// 132-row one 41 to 6.6 (before, one block a piece, each thread waiting for its own loads).
constexpr int TOP_TILE = 128;
template <class T>
__device__ __forceinline__ void dense_rows(int n, int i0, const double* __restrict__ A0, const T* __restrict__ r,
                                           T* __restrict__ z) {
    __shared__ double tile[TOP_TILE][32], rs[TOP_TILE];
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, i = i0 + l;
    const double* A = A0 + i;
    double s = 0.0;
    for (int j0 = 0; j0 < n; j0 += TOP_TILE) {
        if (j0) __syncthreads();
        double a[TOP_TILE / 8];
#pragma unroll
        for (int k = 0; k < TOP_TILE / 8; k++) {
            const int j = j0 + w + 8 * k;
            a[k] = j < n && i < n ? __ldg(A + (int64_t)j * n) : 0.0;
        }
        if (threadIdx.x < TOP_TILE && j0 + (int)threadIdx.x < n) rs[threadIdx.x] = (double)r[j0 + threadIdx.x];
#pragma unroll
        for (int k = 0; k < TOP_TILE / 8; k++) tile[w + 8 * k][l] = a[k];
        __syncthreads();
        if (w == 0) {
            const int m = min(TOP_TILE, n - j0);
#pragma unroll 16
            for (int j = 0; j < m; j++) s = fma(tile[j][l], rs[j], s);
        }
    }
    if (w == 0 && i < n) z[i] = (T)s;
}

// z = Kinv r over each top piece's parts
template <class T>
__global__ void __launch_bounds__(256) k_top_solve(const int32_t* __restrict__ top, const int64_t* __restrict__ pstart,
                                                   const int64_t* __restrict__ kinv_off, const double* __restrict__ kinv,
                                                   const T* __restrict__ r, T* __restrict__ z,
                                                   const int32_t* __restrict__ done) {
    const int p = top[blockIdx.x];
    const int64_t k0 = pstart[p], off = kinv_off[blockIdx.x];
    const int n = (int)(6 * (pstart[p + 1] - k0)), i0 = blockIdx.y * 32;
    if ((done && done[p]) || i0 >= n) return;
    dense_rows<T>(n, i0, kinv + off, r + 6 * k0, z + 6 * k0);
}

// x = A' b, A (n x n) row-major
__global__ void __launch_bounds__(256) k_dense_apply(int n, const double* __restrict__ A, const double* __restrict__ b,
                                                     double* __restrict__ x) {
    dense_rows<double>(n, blockIdx.x * 32, A, b, x);
}

// out[p] = sum over piece p's parts of a.b
template <class T, bool SPLIT>
__global__ void __launch_bounds__(RED_LANES) k_seg_dot(Chunks ch, const T* __restrict__ a, const T* __restrict__ b,
                                                       double* __restrict__ out) {
    extern __shared__ double sm[];
    const int c = red_chunk<SPLIT>(), t = red_lane<SPLIT>(), p = ch.piece[c];
    double s = 0.0, none = 0.0;
    if (!red_run<SPLIT, 2, 8>(
            sm, 6 * ch.lo[c] + t, 6 * ch.lo[c + 1],
            [&](int64_t i, double (&v)[2]) { v[0] = (double)a[i], v[1] = (double)b[i]; },
            [&](const double (&v)[2]) { s = fma(v[0], v[1], s); }))
        return;
    if (red_finish<SPLIT>(ch, c, t, p, s, none)) out[p] = s;
}

// The last power iteration: per piece step = 4/3 / (|w| / |v|) (bodies.rs:174, 187)
template <bool SPLIT>
__global__ void __launch_bounds__(RED_LANES) k_power_step(Chunks ch, const double* __restrict__ w,
                                                          const double* __restrict__ v, double* __restrict__ step) {
    extern __shared__ double sm[];
    const int c = red_chunk<SPLIT>(), t = red_lane<SPLIT>(), p = ch.piece[c];
    double ww = 0.0, vv = 0.0;
    if (!red_run<SPLIT, 2, 8>(
            sm, 6 * ch.lo[c] + t, 6 * ch.lo[c + 1], [&](int64_t i, double (&x)[2]) { x[0] = w[i], x[1] = v[i]; },
            [&](const double (&x)[2]) {
                ww = fma(x[0], x[0], ww);
                vv = fma(x[1], x[1], vv);
            }))
        return;
    if (red_finish<SPLIT>(ch, c, t, p, ww, vv)) step[p] = 4.0 / 3.0 / (sqrt(ww) / sqrt(vv));
}

}  // namespace

template <class T, int WPR>
void launch_split(Context& ctx, int mode, int64_t nrows, const int64_t* rowptr, const int32_t* col, const T* val,
                  const T* x, const T* r, T* y, const T* inv, const double* step, const int32_t* piece,
                  const int32_t* skip_row, const int32_t* done, T* y2) {
    constexpr int RPC = split_warps<T, WPR>() / WPR;
    constexpr int threads = 32 * split_warps<T, WPR>();
    const unsigned g = grid_for(nrows, RPC);
    auto go = [&](auto kernel) {
        kernel<<<g, threads, 0, ctx.stream>>>(nrows, rowptr, col, val, x, r, y, inv, step, piece, skip_row, done, y2);
    };
    switch (mode) {
        case SPMV_Y: go(k_spmv_split<T, SPMV_Y, WPR>); break;
        case SPMV_ADD: go(k_spmv_split<T, SPMV_ADD, WPR>); break;
        case SPMV_RES: go(k_spmv_split<T, SPMV_RES, WPR>); break;
        case SPMV_Y_JACOBI: go(k_spmv_split<T, SPMV_Y_JACOBI, WPR>); break;
        default: go(k_spmv_split<T, SPMV_RES_SMOOTH, WPR>);
    }
    SC_LAUNCH_CK();
}

// Warps a row: half a warp (0) where rows average under 12 blocks; one, unless the rows
// are too few to fill the device twice over and each warp would still stream 16 or more
// blocks (doubling up to 32).
static int warps_per_row(const Context& ctx, int64_t nrows, int64_t nnz) {
    const int64_t target = (int64_t)ctx.sms * 64;  // two waves of 32 warps an SM
    const int64_t avg = nnz / std::max<int64_t>(nrows, 1);
    if (avg < 12) return 0;
    int w = 1;
    while (w < 32 && nrows * w < target && avg >= 32 * w) w *= 2;
    return w;
}

template <class T>
void spmv(Context& ctx, int mode, int64_t nrows, const int64_t* rowptr, const int32_t* col, const T* val, const T* x,
          const T* r, T* y, const T* inv, const double* step, const int32_t* piece, const int32_t* skip_row,
          const int32_t* done, int64_t nnz, T* y2) {
    if (nrows <= 0) return;
    const int wpr = nnz > 0 ? warps_per_row(ctx, nrows, nnz) : 1;
    auto split = [&](auto launch) {
        launch(ctx, mode, nrows, rowptr, col, val, x, r, y, inv, step, piece, skip_row, done, y2);
    };
    switch (wpr) {
        case 2: return split(launch_split<T, 2>);
        case 4: return split(launch_split<T, 4>);
        case 8: return split(launch_split<T, 8>);
        case 16: return split(launch_split<T, 16>);
        case 32: return split(launch_split<T, 32>);
        default: break;
    }
    const unsigned g = grid_for(nrows * (wpr == 0 ? 16 : 32), 256);
    auto go = [&](auto half, auto whole) {
        (wpr == 0 ? half : whole)<<<g, 256, 0, ctx.stream>>>(nrows, rowptr, col, val, x, r, y, inv, step, piece,
                                                             skip_row, done, y2);
    };
    switch (mode) {
        case SPMV_Y: go(k_spmv_half<T, SPMV_Y>, k_spmv<T, SPMV_Y>); break;
        case SPMV_ADD: go(k_spmv_half<T, SPMV_ADD>, k_spmv<T, SPMV_ADD>); break;
        case SPMV_RES: go(k_spmv_half<T, SPMV_RES>, k_spmv<T, SPMV_RES>); break;
        case SPMV_Y_JACOBI: go(k_spmv_half<T, SPMV_Y_JACOBI>, k_spmv<T, SPMV_Y_JACOBI>); break;
        default: go(k_spmv_half<T, SPMV_RES_SMOOTH>, k_spmv<T, SPMV_RES_SMOOTH>);
    }
    SC_LAUNCH_CK();
}

template <class T>
void jacobi(Context& ctx, int64_t n, const T* inv, const T* r, T* x, const double* step, const int32_t* piece,
            const int32_t* skip_row, const int32_t* done) {
    if (n <= 0) return;
    k_jacobi<T><<<grid_for(n, 256), 256, 0, ctx.stream>>>(n, inv, r, x, step, piece, skip_row, done);
    SC_LAUNCH_CK();
}

template <class T>
void top_solve(Context& ctx, const Level& L, const T* r, T* z, const int32_t* done) {
    if (L.top_h.empty()) return;
    int64_t maxn = 0;
    for (int p : L.top_h) maxn = std::max<int64_t>(maxn, 6 * (L.pstart[p + 1] - L.pstart[p]));
    if (maxn <= 0) return;
    const dim3 grid((unsigned)L.top_h.size(), grid_for(maxn, 32));
    k_top_solve<T><<<grid, 256, 0, ctx.stream>>>(L.top.get(), L.pstart_d.get(), L.kinv_off.get(), L.kinv.get(), r, z,
                                                 done);
    SC_LAUNCH_CK();
}

void dense_apply(Context& ctx, int64_t n, const double* A, const double* b, double* x) {
    if (n <= 0) return;
    k_dense_apply<<<grid_for(n, 32), 256, 0, ctx.stream>>>((int)n, A, b, x);
    SC_LAUNCH_CK();
}

// The level's chunks with the context's scratch for their sums (grown here, so never inside
// a capture).
Chunks red_chunks(Context& ctx, const Level& L) {
    const size_t nch = (size_t)std::max<int64_t>(L.nchunks, 1), np = L.pstart.size();
    const size_t sums = 2 * nch + (red_split(L.nchunks) ? 2 * RED_LANES * nch : 0), counts = nch + np;
    if (ctx.red_sums.size() < sums) ctx.red_sums.alloc(sums + 1024, ctx.stream, &ctx.mem);
    if (ctx.red_count.size() < counts) {
        ctx.red_count.alloc(counts + 1024, ctx.stream, &ctx.mem);
        ctx.red_count.zero();
    }
    Chunks ch;
    ch.lo = L.chunk_lo.get();
    ch.piece = L.chunk_piece.get();
    ch.piece_chunk = L.piece_chunk.get();
    ch.part = ctx.red_sums.get();
    ch.lanes = ctx.red_sums.get() + 2 * nch;
    ch.arrived = ctx.red_count.get();
    ch.ticket = ctx.red_count.get() + nch;
    return ch;
}

template <class T>
void seg_dot_t(Context& ctx, const Level& L, const T* a, const T* b, double* out) {
    const int np = (int)L.pstart.size() - 1;
    bool empty = false;  // a piece without parts sums to zero
    for (int p = 0; p < np && !empty; p++) empty = L.pstart[p] == L.pstart[p + 1];
    if (empty) SC_CK(cudaMemsetAsync(out, 0, np * sizeof(double), ctx.stream));
    if (L.nchunks <= 0) return;
    const Chunks ch = red_chunks(ctx, L);
    const unsigned grid = red_grid(L.nchunks);
    if (red_split(L.nchunks))
        k_seg_dot<T, true><<<grid, RED_LANES, red_smem<true>(2), ctx.stream>>>(ch, a, b, out);
    else
        k_seg_dot<T, false><<<grid, RED_LANES, 0, ctx.stream>>>(ch, a, b, out);
    SC_LAUNCH_CK();
}

void power_step(Context& ctx, const Level& L, const double* w, const double* v, double* step) {
    const int np = (int)L.pstart.size() - 1;
    SC_CK(cudaMemsetAsync(step, 0xff, np * sizeof(double), ctx.stream));  // NaN where a piece has no part here
    if (L.nchunks <= 0) return;
    const Chunks ch = red_chunks(ctx, L);
    const unsigned grid = red_grid(L.nchunks);
    if (red_split(L.nchunks))
        k_power_step<true><<<grid, RED_LANES, red_smem<true>(2), ctx.stream>>>(ch, w, v, step);
    else
        k_power_step<false><<<grid, RED_LANES, 0, ctx.stream>>>(ch, w, v, step);
    SC_LAUNCH_CK();
}

void seg_dot(Context& ctx, const Level& L, const double* a, const double* b, double* out) {
    seg_dot_t<double>(ctx, L, a, b, out);
}

#define SC_INST(T)                                                                                                 \
    template void spmv<T>(Context&, int, int64_t, const int64_t*, const int32_t*, const T*, const T*, const T*, T*, \
                          const T*, const double*, const int32_t*, const int32_t*, const int32_t*, int64_t, T*);   \
    template void jacobi<T>(Context&, int64_t, const T*, const T*, T*, const double*, const int32_t*,              \
                            const int32_t*, const int32_t*);                                                       \
    template void top_solve<T>(Context&, const Level&, const T*, T*, const int32_t*);                             \
    template void seg_dot_t<T>(Context&, const Level&, const T*, const T*, double*);
SC_INST(double)
SC_INST(float)

}  // namespace sc
