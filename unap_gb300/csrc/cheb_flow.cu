// The coarse end of a Chebyshev V-cycle in one launch (see cheby.hpp).
//
// From the first tail level down to the coarsest and back, the V-cycle is a
// list of stages: restriction fused with a level's first step, Chebyshev
// steps, residual, the coarsest dense product in column chunks and their
// sums, prolongation.  Every stage writes vectors of its own, filled with
// 0xff bytes before the launch, and a row is computed as soon as the values
// it reads are there (flow_values.cuh), so stages follow one another without
// a launch or a barrier between them.  Warps take tasks from counters in
// stage order, as the sweeps do (flow.cu): the waits end whatever part of the
// grid is resident.  A stage costs 2 to 3 us (a hop of 0.5 to 1, the longest
// row's sum), a launch 3 to 5: V-cycle of a 508,200-cell log-normal hierarchy (Chebyshev on every level)
// 0.454 ms without the tail, 0.374 / 0.364 / 0.355 / 0.388 / 0.485 with it up
// to 12,000 / 30,000 / 60,000 / 120,000 / 250,000 rows; of 4,096,000 cells
// 1.249 and 1.142 ms (60,000).
//
// Each row's arithmetic is the per-step kernels' (cheb_step_kernel,
// residual_kernel, restrict_cheb_zero_kernel, prolong_to_kernel,
// dense_apply_kernel's chunk order): the V-cycle's bits are the same.
//
// Matrix rows take 4 lanes each: levels this small are bound by the chain of
// stages, and a row's entries are then asked for at once.
#include <algorithm>
#include <atomic>

#include "cheby.hpp"
#include "flow.hpp"
#include "flow_values.cuh"

namespace unapgpu {

namespace {

std::atomic<int> g_tailRows{kChebTailRows};

constexpr int kThreads = 128;
constexpr int kStreams = kThreads / 32;
static_assert(kFlowHeader >= kStreams * kFlowCounterBytes, "a counter per stream");
constexpr int G = 4;        // lanes a matrix row
constexpr int RW = 32 / G;  // rows of a matrix task

enum StageType : int { CF_ZERO, CF_STEP, CF_RESIDUAL, CF_RESTRICT, CF_CHUNK, CF_SUM, CF_PROLONG };

template <class T>
struct Stage {
    int type, first;  // first: a chain's first step
    int n, task0;     // rows; first task
    int wait;         // rows of `near`, 0: none
    int pollA;        // a is written in this launch
    Rows<T> A;
    const int* i0;    // children starts, or the prolongation map
    const int* i1;    // children
    const T* a;       // previous iterate, finer residual, coarser result
    const T* b;       // right-hand side (prolongation: own iterate)
    const T* w;       // previous step's correction
    const T* near;    // a vector of the stage before the previous one
    T* x;             // results: iterate, residual, right-hand side ...
    T* y;             // ... and correction / first iterate
    T* copy;          // also written here, for kernels after the launch
    T c1, c2;
};

template <class T>
struct Args {
    const Stage<T>* stage;
    int nStages, nTasks;
    const double* M;   // dense inverse, column-major
    double* part;      // its chunk sums, [chunk][row]
    int nc;
    unsigned* counter;
    WaitBound bound;
};

// the next task of this warp (flow.cu's counters)
__device__ __forceinline__ int take(unsigned* counters)
{
    const unsigned w = threadIdx.x >> 5;
    int t = 0;
    if ((threadIdx.x & 31) == 0)
        t = (int)((atomicAdd(counters + (kFlowCounterBytes / 4) * w, 1u) + 1u) * kStreams + w);
    return t;
}

// one value that another row of this launch writes; all lanes call it
template <class T>
__device__ __forceinline__ T wait_one(const T* p, bool on, int* err)
{
    T v[1] = {T(0)};
    wait_values<T, 1>(on ? 1u : 0u, [&](int) { return p; }, v, err);
    return v[0];
}

// matrix rows: a Chebyshev step or a residual
template <class T, int K>
__device__ __forceinline__ void row_task(const Args<T>& a, const Stage<T>& S, int i, T* pw)
{
    constexpr int W = G * K, P = W + 5;
    const int lane = threadIdx.x & 31, row = lane % RW, g = lane / RW;
    const int r0 = i * RW, r = r0 + row;
    const bool on = r < S.n;
    const int off = ldg(S.A.sliceOff + (r0 >> 5));
    const int w = (ldg(S.A.sliceOff + (r0 >> 5) + 1) - off) / 32;
    const int base = off + (r & 31);
    int len = 0;
    T d = T(1);
    if (on) {
        len = row_len(ldg(S.A.rowInfo + r));
        d = ldg(S.A.diag + r);
    }
    int c[K];
    T v[K], xv[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const bool has = on && k * G + g < w;
        c[k] = has ? ldg(S.A.col + base + 32 * (k * G + g)) : 0;
        v[k] = has ? ldg(S.A.val + base + 32 * (k * G + g)) : T(0);
    }
    const T rD = T(1) / d;
    if (S.wait) wait_near(S.near + (int)((long long)r0 * S.wait / S.n), a.bound);
    // the row's own values: x, b and w, a lane each
    const T* own = g == 0 ? S.a + r : g == 1 ? S.b + r : S.w + r;
    const bool mine = on && (g < 2 || (g == 2 && S.type == CF_STEP && !S.first));
    T acc = T(0), xr = T(0), bb = T(0), wr = T(0);
    for (int j0 = 0;;) {
        unsigned need = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            xv[k] = T(0);
            if (j0 + k * G + g < len) need |= 1u << k;
        }
        T all[K + 1];
        all[K] = T(0);
        if (j0 == 0 && mine) need |= 1u << K;
        wait_values<T, K + 1>(
            need, [&](int k) { return k == K ? own : S.a + c[k]; }, all, a.bound.err);
#pragma unroll
        for (int k = 0; k < K; ++k) pw[row * P + k * G + g] = v[k] * all[k];
        if (j0 == 0) {
            xr = __shfl_sync(0xffffffffu, all[K], row);
            bb = __shfl_sync(0xffffffffu, all[K], row + RW);
            wr = __shfl_sync(0xffffffffu, all[K], row + 2 * RW);
            acc += d * xr;
        }
        __syncwarp();
        if (g == 0) {
            // A x in the reference's order: the diagonal, then the row's faces
            const int m = min(len - j0, W);
            const T* p = pw + row * P;
            T p0 = p[0], p1 = p[1], p2 = p[2], p3 = p[3];
            int j = 0;
            for (; j + 4 <= m; j += 4) {
                // the next four (a row's pitch leaves room for them)
                const T n0 = p[j + 4], n1 = p[j + 5], n2 = p[j + 6], n3 = p[j + 7];
                acc += p0;
                acc += p1;
                acc += p2;
                acc += p3;
                p0 = n0;
                p1 = n1;
                p2 = n2;
                p3 = n3;
            }
            if (j < m) acc += p0;
            if (j + 1 < m) acc += p1;
            if (j + 2 < m) acc += p2;
        }
        __syncwarp();
        j0 += W;
        if (j0 >= w || !__any_sync(0xffffffffu, j0 < len)) break;
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int j = j0 + k * G + g;
            c[k] = j < len ? ldg(S.A.col + base + 32 * j) : 0;
            v[k] = j < len ? ldg(S.A.val + base + 32 * j) : T(0);
        }
    }
    if (!on || g != 0) return;
    if (S.type == CF_RESIDUAL) {
        st_flow(S.x + r, bb - acc);
        return;
    }
    T wi;
    if (S.first)
        wi = rD * (bb - acc) * S.c1;
    else
        wi = S.c1 * wr + S.c2 * rD * (bb - acc);
    const T xi = xr + wi;
    st_flow(S.x + r, xi);
    if (S.y) st_flow(S.y + r, wi);
    if (S.copy) S.copy[r] = xi;
}

// restriction: children in ascending order; CF_ZERO also takes the level's
// first step from x = 0
template <class T>
__device__ __forceinline__ void restrict_task(const Args<T>& a, const Stage<T>& S, int i)
{
    const int r0 = i * 32, r = r0 + (int)(threadIdx.x & 31);
    const bool on = r < S.n;
    int k0 = 0, k1 = 0;
    T d = T(1);
    if (on) {
        k0 = ldg(S.i0 + r);
        k1 = ldg(S.i0 + r + 1);
        if (S.type == CF_ZERO) d = ldg(S.A.diag + r);
    }
    if (S.wait) wait_near(S.near + (int)((long long)r0 * S.wait / S.n), a.bound);
    T acc = T(0);
    for (; __any_sync(0xffffffffu, k0 < k1); k0 += 4) {
        int c[4];
        T v[4];
        unsigned need = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool has = k0 + k < k1;
            c[k] = has ? ldg(S.i1 + k0 + k) : 0;
            v[k] = T(0);
            if (has) need |= 1u << k;
        }
        if (S.pollA) {
            wait_values<T, 4>(need, [&](int k) { return S.a + c[k]; }, v, a.bound.err);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (need >> k & 1u) v[k] = S.a[c[k]];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k0 + k < k1) acc += v[k];
    }
    if (!on) return;
    st_flow(S.x + r, acc);
    if (S.type == CF_ZERO) {
        const T rD = T(1) / d;
        st_flow(S.y + r, rD * acc * S.c1);
    }
}

template <class T>
__global__ void __launch_bounds__(kThreads) cheb_flow_kernel(const __grid_constant__ Args<T> a,
                                                             Gate gate)
{
    if (gate_closed(gate)) return;
    constexpr int K = 8;  // 32 entries a row are loaded before any wait
    __shared__ int task0[kChebTailMaxStages + 1];
    __shared__ T prod[kThreads / 32][RW * (G * K + 5)];
    __shared__ double sb[kThreads / 32][kDenseChunk];
    for (int i = threadIdx.x; i < a.nStages; i += kThreads) task0[i] = a.stage[i].task0;
    if (threadIdx.x == 0) task0[a.nStages] = a.nTasks;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int s = 0;
    for (;;) {
        const int t = __shfl_sync(0xffffffffu, take(a.counter), 0);
        if (t >= a.nTasks) return;
        while (t >= task0[s + 1]) ++s;  // a warp's tasks ascend
        const Stage<T>& S = a.stage[s];
        const int i = t - task0[s];
        if (S.type == CF_STEP || S.type == CF_RESIDUAL) {
            row_task<T, K>(a, S, i, prod[warp]);
        } else if (S.type == CF_ZERO || S.type == CF_RESTRICT) {
            restrict_task<T>(a, S, i);
        } else if (S.type == CF_PROLONG) {
            const int r0 = i * 32, r = r0 + lane;
            const bool on = r < S.n;
            const int c = on ? ldg(S.i0 + r) : 0;
            if (S.wait) wait_near(S.near + (int)((long long)r0 * S.wait / S.n), a.bound);
            T v[2];
            wait_values<T, 2>(on ? 3u : 0u, [&](int k) { return k ? S.a + c : S.b + r; }, v, a.bound.err);
            if (on) st_flow(S.x + r, v[0] + v[1]);
        } else if (S.type == CF_CHUNK) {
            // a column chunk of 32 rows of x = Minv b, summed in ascending
            // order from 0 (dense_apply_kernel)
            const int nb = (a.nc + 31) / 32, q = i / nb, r = (i - q * nb) * 32 + lane;
            const int j0 = q * kDenseChunk, m = min(kDenseChunk, a.nc - j0);
            const double* M = a.M + (size_t)j0 * a.nc + min(r, a.nc - 1);
            double mv[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) mv[k] = k < m ? ldg(M + (size_t)k * a.nc) : 0.0;
            if (S.wait) wait_near(S.near + (int)((long long)j0 * S.wait / S.n), a.bound);
            __syncwarp();
            for (int j = lane; j < kDenseChunk; j += 32) {
                const T b = wait_one<T>(S.a + j0 + j, j < m, a.bound.err);
                sb[warp][j] = (double)b;
            }
            __syncwarp();
            if (r < a.nc) {
                // the next eight columns are loaded while eight are summed
                double p = 0.0;
                double u[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) u[k] = mv[k];
                for (int j = 0; j < m; j += 8) {
                    double nx[8];
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        nx[k] = j + 8 + k < m ? ldg(M + (size_t)(j + 8 + k) * a.nc) : 0.0;
#pragma unroll
                    for (int k = 0; k < 8; ++k) u[k] = u[k] * sb[warp][min(j + k, m - 1)];
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        if (j + k < m) p += u[k];
#pragma unroll
                    for (int k = 0; k < 8; ++k) u[k] = nx[k];
                }
                st_flow(a.part + (size_t)q * a.nc + r, p);
            }
        } else {  // CF_SUM: the chunk sums in chunk order from 0
            const int r = i * 32 + lane;
            const bool on = r < a.nc;
            const int nq = (a.nc + kDenseChunk - 1) / kDenseChunk;
            if (S.wait) wait_near(S.near + (int)((long long)i * 32 * S.wait / S.n), a.bound);
            double t_ = 0.0;
            for (int q0 = 0; q0 < nq; q0 += 4) {
                double v[4];
                const unsigned need = on ? (1u << min(4, nq - q0)) - 1u : 0u;
                wait_values<double, 4>(
                    need, [&](int k) { return a.part + (size_t)(q0 + k) * a.nc + r; }, v, a.bound.err);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (q0 + k < nq) t_ += v[k];
            }
            if (on) st_flow(S.x + r, (T)t_);
        }
    }
}

}  // namespace

int set_cheby_tail_rows(int rows) { return g_tailRows.exchange(std::max(rows, 0)); }
int cheby_tail_rows() { return g_tailRows.load(); }

template <class T>
void ChebFlow<T>::build(const std::vector<ChebFlowLevel<T>>& lev, int deg, const T* rIn, int nc_,
                        const int* cChildStart, const int* cChild, const int* cCmap,
                        const double* Minv, T* result, cudaStream_t s)
{
    static_assert(sizeof(Stage<T>) % 8 == 0, "");
    const int L = (int)lev.size();
    const int nChunks = (nc_ + kDenseChunk - 1) / kDenseChunk;
    nc = nc_;
    M = Minv;
    // vectors: per level b, deg iterates and deg - 1 corrections before, the
    // residual, the prolonged iterate, deg iterates and corrections after;
    // the coarsest b and x; the chunk sums
    size_t bytes = kFlowHeader;
    auto place = [&](size_t count, size_t elem) {
        const size_t at = bytes;
        bytes += (count * elem + 255) / 256 * 256;
        return at;
    };
    struct Off {
        size_t b, r, p;
        std::vector<size_t> x, w, px, pw;
    };
    std::vector<Off> off((size_t)L);
    for (int l = 0; l < L; ++l) {
        const size_t n = (size_t)lev[(size_t)l].A.n;
        Off& o = off[(size_t)l];
        o.b = place(n, sizeof(T));
        o.r = place(n, sizeof(T));
        o.p = place(n, sizeof(T));
        for (int j = 0; j < deg; ++j) {
            o.x.push_back(place(n, sizeof(T)));
            o.w.push_back(j ? place(n, sizeof(T)) : o.x[0]);
            o.px.push_back(place(n, sizeof(T)));
            o.pw.push_back(place(n, sizeof(T)));
        }
    }
    const size_t cb = place((size_t)nc, sizeof(T)), cx = place((size_t)nc, sizeof(T));
    const size_t cp = place((size_t)nc * (size_t)nChunks, sizeof(double));
    arena.alloc(bytes);
    if (!err) err = static_cast<int*>(pinned_block_alloc(64));
    *err = 0;
    auto at = [&](size_t o) { return reinterpret_cast<T*>(arena.p + o); };
    std::vector<Stage<T>> st;
    int tasks = 0;
    const T* lastX = nullptr;  // results of the previous two stages
    const T* prevX = nullptr;
    int lastN = 0, prevN = 0;
    auto add = [&](Stage<T> S, int count) {
        S.task0 = tasks;
        S.near = prevX;
        S.wait = prevX ? prevN : 0;
        tasks += count;
        st.push_back(S);
        prevX = lastX;
        prevN = lastN;
        if (S.type != CF_CHUNK) {
            lastX = S.x;
            lastN = S.n;
        }
    };
    auto chain = [&](int l, bool post) {
        const ChebFlowLevel<T>& V = lev[(size_t)l];
        const Off& o = off[(size_t)l];
        for (int j = post ? 0 : 1; j < deg; ++j) {
            Stage<T> S{};
            S.type = CF_STEP;
            S.first = j == 0;
            S.n = V.A.n;
            S.A = V.A;
            S.a = at(post ? (j ? o.px[(size_t)j - 1] : o.p) : o.x[(size_t)j - 1]);
            S.b = at(o.b);
            S.w = j ? at(post ? o.pw[(size_t)j - 1] : o.w[(size_t)j - 1]) : nullptr;
            S.x = at(post ? o.px[(size_t)j] : o.x[(size_t)j]);
            S.y = j + 1 < deg ? at(post ? o.pw[(size_t)j] : o.w[(size_t)j]) : nullptr;
            S.copy = post && l == 0 && j + 1 == deg ? result : nullptr;
            S.c1 = j ? (T)V.d1[j] : (T)V.Rth;
            S.c2 = j ? (T)V.d2[j] : T(0);
            add(S, div_up(V.A.n, RW));
        }
    };
    for (int l = 0; l < L; ++l) {
        const ChebFlowLevel<T>& V = lev[(size_t)l];
        const Off& o = off[(size_t)l];
        Stage<T> Z{};
        Z.type = CF_ZERO;
        Z.n = V.A.n;
        Z.A = V.A;
        Z.i0 = V.childStart;
        Z.i1 = V.child;
        Z.a = l ? at(off[(size_t)l - 1].r) : rIn;
        Z.pollA = l > 0;
        Z.x = at(o.b);
        Z.y = at(o.x[0]);
        Z.c1 = (T)V.Rth;
        add(Z, div_up(V.A.n, 32));
        chain(l, false);
        Stage<T> R{};
        R.type = CF_RESIDUAL;
        R.n = V.A.n;
        R.A = V.A;
        R.a = at(o.x[(size_t)deg - 1]);
        R.b = at(o.b);
        R.x = at(o.r);
        add(R, div_up(V.A.n, RW));
    }
    {
        Stage<T> C{};
        C.type = CF_RESTRICT;
        C.n = nc;
        C.i0 = cChildStart;
        C.i1 = cChild;
        C.a = at(off[(size_t)L - 1].r);
        C.pollA = 1;
        C.x = at(cb);
        add(C, div_up(nc, 32));
        Stage<T> D{};
        D.type = CF_CHUNK;
        D.n = nc;
        D.a = at(cb);
        add(D, div_up(nc, 32) * nChunks);
        Stage<T> E{};
        E.type = CF_SUM;
        E.n = nc;
        E.x = at(cx);
        add(E, div_up(nc, 32));
    }
    for (int l = L - 1; l >= 0; --l) {
        const ChebFlowLevel<T>& V = lev[(size_t)l];
        const Off& o = off[(size_t)l];
        Stage<T> P{};
        P.type = CF_PROLONG;
        P.n = V.A.n;
        P.i0 = l + 1 < L ? lev[(size_t)l + 1].cmap : cCmap;
        P.a = l + 1 < L ? at(off[(size_t)l + 1].px[(size_t)deg - 1]) : at(cx);
        P.b = at(o.x[(size_t)deg - 1]);
        P.x = at(o.p);
        add(P, div_up(V.A.n, 32));
        chain(l, true);
    }
    nStages = (int)st.size();
    nTasks = tasks;
    part = reinterpret_cast<double*>(arena.p + cp);
    stages.upload(reinterpret_cast<const unsigned char*>(st.data()), st.size() * sizeof(Stage<T>), s);
    int dev = 0, sms = 0;
    UNAP_CK(cudaGetDevice(&dev));
    UNAP_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    grid = std::max(1, std::min(div_up(nTasks, kStreams), kChebTailCtas * sms));
    UNAP_CK(cudaStreamSynchronize(s));
}

template <class T>
void ChebFlow<T>::launch(const Exec& ex, Gate g) const
{
    Args<T> a;
    a.stage = reinterpret_cast<const Stage<T>*>(stages.p);
    a.nStages = nStages;
    a.nTasks = nTasks;
    a.M = M;
    a.part = part;
    a.nc = nc;
    a.counter = reinterpret_cast<unsigned*>(arena.p);
    a.bound = {err, spent};
    UNAP_CK(cudaMemsetAsync(arena.p, 0xff, arena.n, ex.s));
    if (!capturing()) count_launches(1);
    cheb_flow_kernel<T><<<grid, kThreads, 0, ex.s>>>(a, g);
    UNAP_CK(cudaGetLastError());
}

template <class T>
ChebFlow<T>::~ChebFlow()
{
    pinned_block_free(err);
}

template struct ChebFlow<float>;
template struct ChebFlow<double>;

}  // namespace unapgpu
