// Products and residuals over large levels with short rows.
//
// In FP64 such a pass is bound by the FP64 pipe as much as by memory: a row of
// seven entries takes 14 FP64 instructions (8 fused), which at the measured
// 0.525 T/s is 0.45 ms (0.26) for 16.8M rows against 0.27 ms for its bytes.
// spmv_kernel and residual_kernel spent more: a thread a row chains four round
// trips (the row's position, its columns and values, the gathers, the store),
// and a dot product's tree per 256 rows cost 5.6 more instructions a row, a
// fence in every thread and a ticket per 256 rows.  Here a grid that just
// fills the GPU walks over the 32-row slices, a warp a slice: while a warp
// gathers for one slice the next slice's columns, values and row data are on
// their way to its registers and the position of the one after it is known.
// A dot product's block sums are formed for eight blocks at a time.
//
// Measured at 256^3, FP64: fused product with its dot product 852 -> 500 us
// (after a cache flush), product 604 -> 483, residual 688 -> 505; at 100^3
// product 41 -> 34, residual 46 -> 35.  No single unit is then above 60 %:
// gathers a slice earlier (128 registers) gave 1 %, 3, 4 or 5 CTAs of 256
// threads an SM were 0 to 50 % slower.
//
// Per-row arithmetic is row_apply's, bit for bit: the reference's leading
// 0 + D x is D x except where that is -0, so it takes no FP64 instruction.
#include <map>
#include <mutex>

#include "device_common.cuh"
#include "row_stream.hpp"

namespace unapgpu {

namespace {

enum Op : int { OP_SPMV, OP_SPMV_PERM, OP_RESIDUAL };

template <class T>
struct StreamArgs {
    Rows<T> A;
    const T* x;
    const T* b;    // right-hand side, or the vector of the dot product (null: none)
    T* out;
    RSpec red;
    const int* perm;  // OP_SPMV_PERM: where a row's result goes
};

// 0 + v
__device__ __forceinline__ float plus_zero(float v)
{
    return __float_as_uint(v) == 0x80000000u ? 0.0f : v;
}
__device__ __forceinline__ double plus_zero(double v)
{
    return (unsigned long long)__double_as_longlong(v) == 0x8000000000000000ull ? 0.0 : v;
}

// a slice's rows as a warp holds them, a lane a row
template <class T, int K>
struct Held {
    int len, base, w;  // entries, position of entry 0, entries of the slice's longest row
    T d;
    int c[K];
    T v[K];
};

template <class T, int K>
__device__ __forceinline__ void load_slice(const Rows<T>& A, int r, int off, int offNext, Held<T, K>& h)
{
    h.base = off + (r & 31);
    h.w = (offNext - off) >> 5;
    h.len = 0;
    h.d = T(0);
    if (r < A.n) {
        h.len = row_len(lds<true>(A.rowInfo + r));
        h.d = lds<true>(A.diag + r);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        // padding entries have a valid column
        h.c[k] = k < h.w ? lds<true>(A.col + h.base + 32 * k) : 0;
        h.v[k] = k < h.w ? lds<true>(A.val + h.base + 32 * k) : T(0);
    }
}

// The sums over a warp of kHold values a lane, each by warp_sum's tree (lane
// pairs 16 apart, then 8, 4, 2, 1) and so with its bits, in 9 additions
// instead of 40: at each of the first three steps a lane adds for half of the
// values and its partner for the others.  Value lane >> 2's sum is returned.
constexpr int kHold = 8;
__device__ __forceinline__ double warp_sums(double (&v)[kHold])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16, h = 4; h >= 1; o >>= 1, h >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const double theirs = __shfl_xor_sync(0xffffffffu, up ? v[k] : v[k + h], o);
            v[k] = (up ? v[k + h] : v[k]) + theirs;
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}

// block_sum's second tree, over the warps of a 256-thread CTA
__device__ __forceinline__ double warps_sum(const double* w)
{
    static_assert(kBlock == 256);
    return (((w[0] + 0.0) + (w[4] + 0.0)) + ((w[2] + 0.0) + (w[6] + 0.0))) +
           (((w[1] + 0.0) + (w[5] + 0.0)) + ((w[3] + 0.0) + (w[7] + 0.0)));
}

// A product's dot product has the bits of a thread a row and a CTA per 256
// rows: a CTA's warps are always at the slices of one such block, and after
// kHold blocks their partial sums are formed, all at once, by the same trees.
template <class T, int K, int OP, bool FM, bool DOT>
__global__ void __launch_bounds__(kBlock)
    row_stream_kernel(const __grid_constant__ StreamArgs<T> a, Gate g)
{
    if (gate_closed(g)) return;
    const int lane = threadIdx.x & 31;
    const int nSlices = (a.A.n + 31) >> 5;
    const int step = (int)(gridDim.x * (kBlock / 32));
    int s = (int)(blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5));
    const int* so = a.A.sliceOff;
    Held<T, K> cur, nxt;
    cur.w = 0;
    int o0 = 0, o1 = 0;  // bounds of the next slice
    if (s < nSlices) {
        load_slice<T, K>(a.A, 32 * s + lane, ldg(so + s), ldg(so + s + 1), cur);
        if (s + step < nSlices) {
            o0 = ldg(so + s + step);
            o1 = ldg(so + s + step + 1);
        }
    }
    __shared__ double prod[DOT ? kHold : 1][DOT ? kBlock : 1];
    __shared__ double sums[2][kHold][kBlock / 32];
    int held = 0, buf = 0;
    const int nBlocks = (a.A.n + kBlock - 1) / kBlock;
    for (int blk = blockIdx.x; blk < nBlocks; blk += gridDim.x, s += step) {
        const int r = 32 * s + lane;
        const bool on = r < a.A.n;
        int to = r;
        T xv[K], xr = T(0), bb = T(0);
        if (on) {
            xr = ldg(a.x + r);
            if (a.b) bb = ldg(a.b + r);
            if (OP == OP_SPMV_PERM) to = lds<true>(a.perm + r);
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
            xv[k] = k < cur.w ? ldg(a.x + cur.c[k]) : T(0);
        const int s1 = s + step;
        if (s1 < nSlices) {
            load_slice<T, K>(a.A, 32 * s1 + lane, o0, o1, nxt);
            if (s1 + step < nSlices) {
                o0 = ldg(so + s1 + step);
                o1 = ldg(so + s1 + step + 1);
            }
        } else {
            nxt.w = 0;
        }
        // the reference's order: 0, + diag x, then the row's faces
        T acc = FM ? cur.d * xr : plus_zero(cur.d * xr);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (k >= cur.w) break;
            if (k < cur.len) {
                if constexpr (FM)
                    acc = fma(cur.v[k], xv[k], acc);
                else
                    acc += cur.v[k] * xv[k];
            }
        }
        // rows longer than K entries
        for (int j0 = K; j0 < cur.w; j0 += 4) {
            int c[4];
            T v[4], y[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool has = j0 + k < cur.len;
                c[k] = has ? lds<true>(a.A.col + cur.base + 32 * (j0 + k)) : 0;
                v[k] = has ? lds<true>(a.A.val + cur.base + 32 * (j0 + k)) : T(0);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                y[k] = j0 + k < cur.len ? ldg(a.x + c[k]) : T(0);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (j0 + k < cur.len) {
                    if constexpr (FM)
                        acc = fma(v[k], y[k], acc);
                    else
                        acc += v[k] * y[k];
                }
        }
        if (on) {
            if constexpr (OP == OP_RESIDUAL)
                a.out[r] = bb - acc;
            else
                a.out[to] = acc;
        }
        if constexpr (DOT) {
            double v = 0.0;
            if (on) v = FM ? fma((double)acc, (double)bb, 0.0) : 0.0 + (double)acc * (double)bb;
            prod[held][threadIdx.x] = v;
            if (++held == kHold || blk + (int)gridDim.x >= nBlocks) {
                double t[kHold];
#pragma unroll
                for (int k = 0; k < kHold; ++k) t[k] = k < held ? prod[k][threadIdx.x] : 0.0;
                const double sum = warp_sums(t);
                if (!(lane & 3)) sums[buf][lane >> 2][threadIdx.x >> 5] = sum;
                __syncthreads();
                if ((int)threadIdx.x < held)
                    a.red.blockPart[blk - (held - 1 - (int)threadIdx.x) * (int)gridDim.x] =
                        warps_sum(sums[buf][threadIdx.x]);
                buf ^= 1;
                held = 0;
            }
        }
        cur = nxt;
    }
    if constexpr (DOT) {
        __threadfence();
        __syncthreads();
        reduce_partials<1>(nBlocks, (int)gridDim.x, a.red,
                           [&](const double (&t)[1]) { apply_fin(a.red.st, a.red.fin, t, 1); });
    }
}

// CTAs of a kernel the current device holds at once
int resident(const void* f)
{
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, int> known;
    int dev = 0;
    UNAP_CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    int& n = known[{dev, f}];
    if (!n) {
        int sms = 0, per = 0;
        UNAP_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        UNAP_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, f, kBlock, 0));
        n = std::max(1, sms * per);
    }
    return n;
}

template <class T, int OP, bool FM, bool DOT>
void launch(const Exec& ex, const StreamArgs<T>& a, Gate g)
{
    auto f = row_stream_kernel<T, 8, OP, FM, DOT>;
    if (!capturing()) count_launches(1);
    f<<<std::min(div_up(a.A.n, kBlock), resident((const void*)f)), kBlock, 0, ex.s>>>(a, g);
}

}  // namespace

template <class T>
bool row_streams(const Rows<T>& A, const RSpec& red)
{
    return !A.wide && A.n >= (sizeof(T) == 8 ? kStreamRows64 : kStreamRows32) &&
           (!red.blockPart || red.maxBlocks >= div_up(A.n, kBlock));
}

template <class T>
void stream_spmv(const Exec& ex, const Rows<T>& A, const T* x, T* y, const T* dotWith, RSpec red,
                 Gate g, bool fused)
{
    StreamArgs<T> a{A, x, red.blockPart ? dotWith : nullptr, y, red};
    if (a.b)
        fused ? launch<T, OP_SPMV, true, true>(ex, a, g) : launch<T, OP_SPMV, false, true>(ex, a, g);
    else
        fused ? launch<T, OP_SPMV, true, false>(ex, a, g)
              : launch<T, OP_SPMV, false, false>(ex, a, g);
}

template <class T>
void stream_spmv_reference(const Exec& ex, const Rows<T>& A, const int* perm, const T* x, T* y)
{
    StreamArgs<T> a{A, x, nullptr, y, RSpec{}, perm};
    launch<T, OP_SPMV_PERM, false, false>(ex, a, Gate{});
}

template <class T>
void stream_residual(const Exec& ex, const Rows<T>& A, const T* x, const T* b, T* r, Gate g)
{
    StreamArgs<T> a{A, x, b, r, RSpec{}};
    launch<T, OP_RESIDUAL, false, false>(ex, a, g);
}

#define UNAP_STREAM_INST(T)                                                                       \
    template bool row_streams<T>(const Rows<T>&, const RSpec&);                                   \
    template void stream_spmv<T>(const Exec&, const Rows<T>&, const T*, T*, const T*, RSpec, Gate, \
                                 bool);                                                           \
    template void stream_spmv_reference<T>(const Exec&, const Rows<T>&, const int*, const T*, T*); \
    template void stream_residual<T>(const Exec&, const Rows<T>&, const T*, const T*, T*, Gate);
UNAP_STREAM_INST(float)
UNAP_STREAM_INST(double)
#undef UNAP_STREAM_INST

}  // namespace unapgpu
