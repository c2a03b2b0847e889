// Wavefront sweeps as one launch (see flow.hpp).
//
// A sweep's rows are cut into tasks of at most 32 rows, one warp each: rows
// of one SELL slice and of one wavefront, so a task's rows are independent.
// Warps take tasks from a counter in dependency order (forward: ascending
// rows, backward: descending).  A task's rows depend only on rows of tasks
// taken before it, by warps that are running or done, so whatever part of
// the grid is resident, the waits end: no co-residency is assumed.
//
// A row waits for its neighbours by value.  The output vector is filled with
// 0xff bytes before the launch (a NaN that no row writes: a result with that
// pattern is written as the default NaN), a row's value is one 4- or 8-byte
// relaxed store, and a reader loads until it sees something else.  The store
// carries its own flag, so no fence, barrier or launch stands between two
// wavefronts: a dependent row costs one store-to-load hop through L2 (0.33
// us) and its own arithmetic, where a launch per wavefront cost 3 to 6 us.
// Old and new values live in different vectors, so no row overwrites what
// another still reads, and several sweeps run in one launch, each following
// the one before by its own waits.
//
// Every wait is bounded (WaitBound): one that runs out, or that sees that
// another wait of the same ring did, goes on with what it has, and the host
// turns the ring's error word into an error (FlowRing::check).
#include <algorithm>

#include "flow.hpp"
#include "flow_values.cuh"

namespace unapgpu {

namespace {

constexpr int kFlowThreads = 128;
constexpr int kStreams = kFlowThreads / 32;  // a task counter for each warp of a CTA
static_assert(kFlowHeader >= kStreams * kFlowCounterBytes, "a counter per stream");

// The next task of this warp.  Warp w of every CTA takes the tasks w, w +
// kStreams, ... from a counter of its own (starting at -1).  As every CTA
// serves every counter, whichever CTAs are resident, no task is left behind.
// One counter hands out a task every 0.65 ns at best, and eight that share
// an L2 slice no more (0.60 ns, 32 bytes apart); 4 KB apart they give one
// every 0.09 ns.
__device__ __forceinline__ int take(unsigned* counters)
{
    const unsigned w = threadIdx.x >> 5;
    int t = 0;
    if ((threadIdx.x & 31) == 0)
        t = (int)((atomicAdd(counters + (kFlowCounterBytes / 4) * w, 1u) + 1u) * kStreams + w);
    return t;
}

template <class T>
struct GsArgs {
    Rows<T> A;
    const int4* task;
    const int2* near;
    int nTasks, nSweeps, firstFromZero;
    const T* in;
    T* out;         // sweep s writes out + s * stride ...
    long long stride;
    T* last;        // ... and the last one here
    T* copy;        // and here, or null,
    const int* copyAt;  // row r at copyAt[r] if given
    const T* b;
    unsigned* counter;
    WaitBound bound;
};

// G lanes a row, K entries a lane, so that a row is loaded whole before its
// turn and its neighbours are asked for at once; with G > 1 the products meet
// in shared memory and one lane takes their ordered sum (a chain of FP64
// additions of 32 ns each on this GPU).  Lane i + (32 / G) g of the warp
// holds entries g, g + G, ... of row i of the task: the lanes of one g read
// consecutive rows.
template <class T, int G, int K, bool BWD>
__global__ void __launch_bounds__(kFlowThreads)
    flow_gs_kernel(const __grid_constant__ GsArgs<T> a, Gate gate)
{
    if (gate_closed(gate)) return;
    constexpr int RW = 32 / G;      // rows of a task
    constexpr int W = G * K;        // entries of a row held at once
    constexpr int P = W + 5;        // row pitch of the products
    __shared__ T prod[kFlowThreads / 32][G == 1 ? 1 : RW * P];
    T* pw = prod[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    const int row = lane % RW, g = lane / RW;
    const int total = a.nTasks * a.nSweeps;
    for (;;) {
        const int t = __shfl_sync(0xffffffffu, take(a.counter), 0);
        if (t >= total) return;
        const int s = a.nSweeps == 1 ? 0 : t / a.nTasks;
        int q = t - s * a.nTasks;
        if (BWD) q = a.nTasks - 1 - q;
        const int4 D = ldg(a.task + q);
        const int2 nr = ldg(a.near + q);
        const int r = D.x + row;
        const bool on = row < D.y;
        T* out = s == a.nSweeps - 1 ? a.last : a.out + s * a.stride;
        const T* in = s == 0 ? a.in : a.out + (s - 1) * a.stride;
        const int base = D.z + row;
        int info = 0;
        T d = T(1), acc = T(0);
        if (on) {
            info = ldg(a.A.rowInfo + r);
            d = ldg(a.A.diag + r);
            acc = __ldcg(a.b + r);
        }
        int c[K];
        T v[K], xv[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const bool has = on && k * G + g < D.w;
            c[k] = has ? ldg(a.A.col + base + 32 * (k * G + g)) : 0;
            v[k] = has ? ldg(a.A.val + base + 32 * (k * G + g)) : T(0);
        }
        const int nLow = row_low(info);
        const int jEnd = !BWD && s == 0 && a.firstFromZero ? nLow : row_len(info);
        if ((BWD ? nr.y : nr.x) >= 0) wait_near(out + (BWD ? nr.y : nr.x), a.bound);
        for (int j0 = 0;;) {
            unsigned need = 0;
            auto at = [&](int k) {
                const int j = j0 + k * G + g;
                return ((BWD ? j >= nLow : j < nLow) ? (const T*)out : in) + c[k];
            };
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int j = j0 + k * G + g;
                xv[k] = T(0);
                if (j < jEnd) {
                    if ((BWD ? j >= nLow : j < nLow) || s > 0)
                        need |= 1u << k;
                    else
                        xv[k] = *at(k);
                }
            }
            wait_values<T, K>(need, at, xv, a.bound.err);
            if (G == 1) {
#pragma unroll
                for (int k = 0; k < K; ++k) xv[k] = v[k] * xv[k];
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    if (j0 + k >= D.w) break;
                    const T less = acc - xv[k];
                    acc = j0 + k < jEnd ? less : acc;
                }
            } else {
#pragma unroll
                for (int k = 0; k < K; ++k) pw[row * P + k * G + g] = v[k] * xv[k];
                __syncwarp();
            }
            if (G > 1 && g == 0) {
                // the reference's order: entry after entry
                const int m = min(jEnd - j0, W);
                const T* p = pw + row * P;
                T p0 = p[0], p1 = p[1], p2 = p[2], p3 = p[3];
                int j = 0;
                for (; j + 4 <= m; j += 4) {
                    // the next four (a row's pitch leaves room for them)
                    const T n0 = p[j + 4], n1 = p[j + 5], n2 = p[j + 6], n3 = p[j + 7];
                    acc -= p0;
                    acc -= p1;
                    acc -= p2;
                    acc -= p3;
                    p0 = n0;
                    p1 = n1;
                    p2 = n2;
                    p3 = n3;
                }
                if (j < m) acc -= p0;
                if (j + 1 < m) acc -= p1;
                if (j + 2 < m) acc -= p2;
            }
            if (G > 1) __syncwarp();
            j0 += W;
            if (j0 >= D.w || !__any_sync(0xffffffffu, j0 < jEnd)) break;
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const int j = j0 + k * G + g;
                c[k] = j < jEnd ? ldg(a.A.col + base + 32 * j) : 0;
                v[k] = j < jEnd ? ldg(a.A.val + base + 32 * j) : T(0);
            }
        }
        if (on && g == 0) {
            acc = acc / d;
            st_flow(out + r, acc);
            if (a.copy && s == a.nSweeps - 1)
                a.copy[a.copyAt ? ldg(a.copyAt + r) : r] = acc;
        }
    }
}

// d_c = D_c - sum over lower-side faces (asc) of (c1 c2) / d_l
// (lduDICPrecond.cpp:15-42, lduDILUPrecond.cpp:15-43), rD = 1 / d, and every
// entry times its row's rD: the first product of the sweeps' rD coef w, taken
// once here instead of in every application (7 FP64 operations a 7-point row
// and sweep instead of 10, on a pipe of 0.525 T operations/s).  c2 is also
// the lower-side coefficient of the forward sweep.
template <int CK>
__global__ void __launch_bounds__(kFlowThreads)
    flow_factor_kernel(Rows<double> A, const int4* task, const int2* near, int nTasks,
                       const double* c1, const double* c2, double* d, double* rD, double* f,
                       unsigned* counter, WaitBound bound)
{
    const int lane = threadIdx.x & 31;
    for (;;) {
        const int q = __shfl_sync(0xffffffffu, take(counter), 0);
        if (q >= nTasks) return;
        const int4 D = ldg(task + q);
        const int wait = ldg(near + q).x;
        const int r = D.x + lane;
        const bool on = lane < D.y;
        const int base = D.z + lane;
        int len = 0, nLow = 0;
        double acc = 1.0;
        if (on) {
            const int info = ldg(A.rowInfo + r);
            len = row_len(info);
            nLow = row_low(info);
            acc = ldg(A.diag + r);
        }
        const int most = __reduce_max_sync(0xffffffffu, nLow);
        for (int j0 = 0; j0 < most; j0 += CK) {
            int c[CK];
            double v[CK], xv[CK];
            unsigned need = 0;
#pragma unroll
            for (int k = 0; k < CK; ++k) {
                const int e = base + 32 * (j0 + k);
                const bool has = j0 + k < nLow;
                c[k] = has ? ldg(A.col + e) : 0;
                // 1 / 1 where there is no entry: one lane's numerator of 0 sends
                // its warp through the division's slow path, which cost half of
                // a 61x97x43 factor's time (169 -> 86 us)
                v[k] = has ? ldg(c1 + e) * ldg(c2 + e) : 1.0;
                xv[k] = 1.0;
                if (has) need |= 1u << k;
            }
            if (j0 == 0 && wait >= 0) wait_near(d + wait, bound);
            wait_values<double, CK>(need, [&](int k) { return (const double*)d + c[k]; }, xv,
                                    bound.err);
#pragma unroll
            for (int k = 0; k < CK; ++k)
                if (j0 + k < most) xv[k] = v[k] / xv[k];
#pragma unroll
            for (int k = 0; k < CK; ++k) {
                if (j0 + k >= most) break;
                const double less = acc - xv[k];
                acc = j0 + k < nLow ? less : acc;
            }
        }
        if (on) {
            st_flow(d + r, acc);
            const double rd = 1.0 / acc;
            rD[r] = rd;
            for (int j = 0; j < len; ++j) {
                const int e = base + 32 * j;
                f[e] = rd * (j < nLow ? ldg(c2 + e) : ldg(A.val + e));
            }
        }
    }
}

struct DicArgs {
    Rows<double> A;
    const int4* task;
    const int2* near;
    int nTasks;
    const double* f;
    const double* rD;
    const double* r;
    double* wf;    // forward sweep's vector
    double* w;
    double* part;  // partial of w.r per task, or null
    unsigned* counter;
    WaitBound bound;
};

// w = M^-1 r (lduDICPrecond.cpp:45-77, lduDILUPrecond.cpp:46-86): the forward
// sweep's tasks, then the backward sweep's.  forward: wf_c = rD_c r_c, then
// wf_c -= (rD_c coef) wf_l over the lower entries in face order; backward:
// w_c = wf_c, then w_c -= (rD_c upper) w_u over the upper entries from the
// last (DIC's face loop in reverse).  Bound by the chain of wavefronts (a
// hop and up to four FP64 operations each) up to some 10^5 rows, by the FP64
// pipe above.
template <int CK>
__global__ void __launch_bounds__(kFlowThreads) flow_dic_kernel(const __grid_constant__ DicArgs a,
                                                                Gate g)
{
    if (gate_closed(g)) return;
    const int lane = threadIdx.x & 31;
    const Rows<double>& A = a.A;
    for (;;) {
        const int t = __shfl_sync(0xffffffffu, take(a.counter), 0);
        if (t >= 2 * a.nTasks) return;
        const bool bwd = t >= a.nTasks;
        const int q = bwd ? 2 * a.nTasks - 1 - t : t;
        const int4 D = ldg(a.task + q);
        const int2 nr = ldg(a.near + q);
        const int r = D.x + lane;
        const bool on = lane < D.y;
        // entry k of the sweep is entry first + k * step of the storage
        int cnt = 0, first = 0;
        const int step = bwd ? -32 : 32;
        double acc = 0.0, rr = 0.0;
        if (on) {
            const int info = ldg(A.rowInfo + r);
            const int len = row_len(info), nLow = row_low(info);
            const int base = D.z + lane;
            cnt = bwd ? len - nLow : nLow;
            first = bwd ? base + 32 * (len - 1) : base;
            rr = __ldcg(a.r + r);
            if (!bwd) acc = ldg(a.rD + r) * rr;
        }
        const int most = __reduce_max_sync(0xffffffffu, cnt);
        double* out = bwd ? a.w : a.wf;
        const int wait = bwd ? nr.y : nr.x;
        int j0 = 0;
        do {
            // slot CK is the backward sweep's own starting value
            int c[CK];
            double v[CK], xv[CK + 1];
            unsigned need = 0;
#pragma unroll
            for (int k = 0; k < CK; ++k) {
                const int e = first + step * (j0 + k);
                const bool has = j0 + k < cnt;
                c[k] = has ? ldg(A.col + e) : 0;
                v[k] = has ? ldg(a.f + e) : 0.0;
                xv[k] = 0.0;
                if (has) need |= 1u << k;
            }
            xv[CK] = 0.0;
            if (bwd && on && j0 == 0) need |= 1u << CK;
            if (j0 == 0 && wait >= 0) wait_near(out + wait, a.bound);
            wait_values<double, CK + 1>(
                need, [&](int k) { return k == CK ? a.wf + r : (const double*)out + c[k]; }, xv,
                a.bound.err);
            if (bwd && j0 == 0) acc = xv[CK];
#pragma unroll
            for (int k = 0; k < CK; ++k) {
                if (j0 + k >= most) break;
                xv[k] = v[k] * xv[k];
            }
#pragma unroll
            for (int k = 0; k < CK; ++k) {
                if (j0 + k >= most) break;
                const double less = acc - xv[k];
                acc = j0 + k < cnt ? less : acc;
            }
            j0 += CK;
        } while (j0 < most);
        if (on) st_flow(out + r, acc);
        if (bwd && a.part) {
            const double s = warp_sum(on ? acc * rr : 0.0);
            if (lane == 0) a.part[q] = s;
        }
    }
}

__global__ void __launch_bounds__(kBlock) flow_sum_kernel(int n, const double* __restrict__ part,
                                                          RSpec red, Gate g)
{
    if (gate_closed(g)) return;
    double v[1] = {0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        v[0] += part[i];
    reduce_launch<1>(v, red, [&](const double (&t)[1]) { apply_fin(red.st, red.fin, t, 1); });
}

void tick()
{
    if (!capturing()) count_launches(1);
}

int sm_count()
{
    static int cached = 0;
    if (!cached) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cached = n > 0 ? n : 152;
    }
    return cached;
}

// fills in where a task's slice starts and how many entries its rows hold
__global__ void task_slices_kernel(int n, const int* __restrict__ sliceOff, int4* task)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int r = task[i].x;
    const int o = sliceOff[r >> 5];
    task[i].z = o + (r & 31);
    task[i].w = (sliceOff[(r >> 5) + 1] - o) / 32;
}

// Lanes a row of a Gauss-Seidel sweep.  A row is one ordered sum: with a lane
// a row its entries' loads wait for one another in chunks, with more lanes
// they are all in flight at once, but a warp holds fewer rows.  Rows of 8 or
// fewer entries fit one lane.  One sweep of the levels of a 128^3 Laplacian's
// hierarchy, us at 1 / 4 / 8 lanes: FP64, 453,513 rows 127 / 184 / -, 215,841
// rows 161 / 151 / 184, 103,381 rows 166 / 147 / 123, 23,973 rows 149 / 119 /
// 96, 2,718 rows 127 / 95 / 69; FP32, 965,724 rows 55 / 86 / -, 453,513 rows
// 67 / 54 / -, 103,381 rows 93 / 54 / 70, 23,973 rows 86 / 53 / 64.
int sweep_lanes(int n, double len, bool fp64)
{
    if (len <= 8.5) return 1;
    if (fp64 && n <= 150000) return 8;
    return n <= (fp64 ? 300000 : 600000) ? 4 : 1;
}

int flow_grid(long long tasks)
{
    constexpr int W = kFlowThreads / 32;
    return (int)std::max(1LL, std::min((tasks + W - 1) / W, 12LL * sm_count()));
}

}  // namespace

void flow_tasks(Level& L, cudaStream_t s)
{
    if (!L.sweepable) return;
    const double len = L.n ? 2.0 * L.nf / L.n : 0.0;
    // every table's tasks, then its near rows two an int4: one allocation and one
    // copy a level (making an MG hierarchy of 1,728 cells took 1.17 ms with two
    // allocations a table and a synchronization after each, 1.05 with this)
    std::vector<int4> all;
    size_t first[3] = {};
    for (SweepTasks& S : L.tasks) {
        if (S.lanes > 1 && S.lanes != sweep_lanes(L.n, len, true) &&
            S.lanes != sweep_lanes(L.n, len, false))
            continue;
        const int rows = 32 / S.lanes;
        std::vector<int2> near;
        near.reserve((size_t)(L.n / rows + L.nWave + 2));
        const size_t at = first[&S - L.tasks] = all.size();
        for (int w = 0; w < L.nWave; ++w) {
            const int r0 = L.waveStart[(size_t)w], r1 = L.waveStart[(size_t)w + 1];
            // a row at the same relative place of wavefront v
            auto beside = [&](int v, int r) {
                if (v < 0 || v >= L.nWave) return -1;
                const int a = L.waveStart[(size_t)v], m = L.waveStart[(size_t)v + 1] - a;
                return m > 0 ? a + (int)((long long)(r - r0) * m / (r1 - r0)) : -1;
            };
            for (int r = r0; r < r1;) {
                const int e = std::min(r1, (r / rows + 1) * rows);
                all.push_back(make_int4(r, e - r, 0, 0));
                near.push_back(make_int2(beside(w - 2, r), beside(w + 2, r)));
                r = e;
            }
        }
        S.n = (int)(all.size() - at);
        near.resize((near.size() + 1) / 2 * 2);
        for (size_t i = 0; i < near.size(); i += 2)
            all.push_back(make_int4(near[i].x, near[i].y, near[i + 1].x, near[i + 1].y));
    }
    L.taskMem.upload(all, s);
    for (SweepTasks& S : L.tasks) {
        if (!S.n) continue;
        S.task = L.taskMem.p + first[&S - L.tasks];
        S.near = reinterpret_cast<int2*>(S.task + S.n);
        task_slices_kernel<<<div_up(S.n, 256), 256, 0, s>>>(S.n, L.d_sliceOff.p, S.task);
        UNAP_CK(cudaGetLastError());
    }
    UNAP_CK(cudaStreamSynchronize(s));  // the host's copy dies here
}

template <class T, bool BWD>
static void launch_gs(const Exec& ex, int wide, int lanes, const GsArgs<T>& a, Gate g)
{
    const int grid = flow_grid((long long)a.nTasks * a.nSweeps);
    if (lanes == 8)
        flow_gs_kernel<T, 8, 4, BWD><<<grid, kFlowThreads, 0, ex.s>>>(a, g);
    else if (lanes == 4)
        flow_gs_kernel<T, 4, 6, BWD><<<grid, kFlowThreads, 0, ex.s>>>(a, g);
    else if (wide)
        flow_gs_kernel<T, 1, 16, BWD><<<grid, kFlowThreads, 0, ex.s>>>(a, g);
    else
        flow_gs_kernel<T, 1, 8, BWD><<<grid, kFlowThreads, 0, ex.s>>>(a, g);
}

template <class T>
T* flow_gs(const Exec& ex, const Level& L, const Rows<T>& A, const FlowRing& ring, const T* in,
           const T* b, int nSweeps, bool backward, bool xIsZero, T* last, T* copy, Gate g,
           const int* copyAt)
{
    const int lanes = L.n ? sweep_lanes(L.n, 2.0 * L.nf / L.n, sizeof(T) == 8) : 1;
    const SweepTasks& S = L.tasks[lanes == 8 ? 2 : lanes == 4 ? 1 : 0];
    T* cur = const_cast<T*>(in);
    const size_t vecBytes = (size_t)L.n * sizeof(T);
    for (int done = 0; done < nSweeps;) {
        const int h = ring.other(cur);
        const int m = std::min(nSweeps - done, ring.sweeps);
        const bool end = done + m == nSweeps;
        GsArgs<T> a;
        a.A = A;
        a.task = S.task;
        a.near = S.near;
        a.nTasks = S.n;
        a.nSweeps = m;
        a.firstFromZero = done == 0 && xIsZero ? 1 : 0;
        a.in = cur;
        a.out = reinterpret_cast<T*>(ring.vec(h, 0));
        a.stride = (long long)(ring.stride / sizeof(T));
        a.last = end && last ? last : reinterpret_cast<T*>(ring.vec(h, m - 1));
        a.copy = end ? copy : nullptr;
        a.copyAt = copyAt;
        a.b = b;
        a.counter = ring.counter(h);
        a.bound = ring.bound();
        const int own = end && last ? m - 1 : m;  // vectors of the ring this launch writes
        UNAP_CK(cudaMemsetAsync(ring.counter(h), 0xff, kFlowHeader + ring.stride * (size_t)own, ex.s));
        if (own < m) UNAP_CK(cudaMemsetAsync(last, 0xff, vecBytes, ex.s));
        tick();
        if (backward)
            launch_gs<T, true>(ex, A.wide, lanes, a, g);
        else
            launch_gs<T, false>(ex, A.wide, lanes, a, g);
        UNAP_CK(cudaGetLastError());
        cur = a.last;
        done += m;
    }
    return cur;
}

template float* flow_gs<float>(const Exec&, const Level&, const Rows<float>&, const FlowRing&,
                               const float*, const float*, int, bool, bool, float*, float*,
                               Gate, const int*);
template double* flow_gs<double>(const Exec&, const Level&, const Rows<double>&, const FlowRing&,
                                 const double*, const double*, int, bool, bool, double*, double*,
                                 Gate, const int*);

void flow_dic_factor(const Exec& ex, const Level& L, bool dilu, DicFlow& D)
{
    if (L.n <= 0) return;
    Rows<double> A = rows64(L);
    // DIC: upper * upper; DILU: upper * lower.  On the lower side of a row the
    // face's upper coefficient is valT and its lower coefficient is val; the
    // forward sweep reads upper (DIC) or lower (DILU) there.
    const double* c1 = A.valT;
    const double* c2 = dilu ? A.val : A.valT;
    double* d = reinterpret_cast<double*>(D.ring.vec(0, 0));
    UNAP_CK(cudaMemsetAsync(D.ring.counter(0), 0xff, kFlowHeader + D.ring.stride, ex.s));
    tick();
    flow_factor_kernel<8><<<flow_grid(L.tasks[0].n), kFlowThreads, 0, ex.s>>>(
        A, L.tasks[0].task, L.tasks[0].near, L.tasks[0].n, c1, c2, d, D.rD.p, D.f.p,
        D.ring.counter(0), D.ring.bound());
    UNAP_CK(cudaGetLastError());
}

void flow_dic_apply(const Exec& ex, const Level& L, const DicFlow& D, const double* r, double* w,
                    const RedPool* pool, int site, KState* st, int fin, Gate g)
{
    if (L.n <= 0) return;
    DicArgs a;
    a.A = rows64(L);
    a.task = L.tasks[0].task;
    a.near = L.tasks[0].near;
    a.nTasks = L.tasks[0].n;
    a.f = D.f.p;
    a.rD = D.rD.p;
    a.r = r;
    a.wf = reinterpret_cast<double*>(D.ring.vec(0, 0));
    a.w = w;
    a.part = pool ? D.part.p : nullptr;
    a.counter = D.ring.counter(0);
    a.bound = D.ring.bound();
    UNAP_CK(cudaMemsetAsync(a.counter, 0xff, kFlowHeader + D.ring.stride, ex.s));
    UNAP_CK(cudaMemsetAsync(w, 0xff, (size_t)L.n * sizeof(double), ex.s));
    tick();
    flow_dic_kernel<8><<<flow_grid(2LL * L.tasks[0].n), kFlowThreads, 0, ex.s>>>(a, g);
    if (pool) {
        tick();
        flow_sum_kernel<<<ex.grid(div_up(L.tasks[0].n, 4)), kBlock, 0, ex.s>>>(
            L.tasks[0].n, D.part.p, pool->site(site, st, fin), g);
    }
    UNAP_CK(cudaGetLastError());
}

void small_sweeps(SmallSystem& S, const Level& L, const DicFlow& D)
{
    S.rD = D.rD.p;
    S.f = D.f.p;
    S.task = L.tasks[0].task;
    S.near = L.tasks[0].near;
    S.nTasks = L.tasks[0].n;
    S.err = D.ring.err;
    S.spent = D.ring.spent;
}

}  // namespace unapgpu
