// batched_cluster.cu -- independent Jacobi-PCG solves from shared memory: one
// CTA, or one cluster of up to 16 CTAs, per system.
//
// The kernels of batched_kernels.cu give a system one CTA and stream it from
// L2 and HBM in every iteration.  With thousands of systems that keeps the FP64
// pipes 80 % busy.  With few, or with a few long ones, the batch takes as long
// as its longest system on one SM: 20,000 rows at 2 FP64 FMAs per clock are 50
// us per iteration and up.  Here a system's rows are spread over as many CTAs
// as hold its matrix and p in shared memory; thread t owns rows t, t + NT, ...
// of its CTA in the product and in the updates, so r, x, J, z and Ap never
// leave its registers, and an iteration touches no global memory.  CTAs gather
// p from one another through distributed shared memory where a row reaches
// outside its CTA.  The sums of the CTAs meet by st.async, which counts itself
// at the receiver's mbarrier: no barrier of the cluster, one CTA barrier on
// either side.  One barrier of the cluster per iteration publishes p.
//
// What bounds it: the chain of dependent steps (an FP64 add 64 cycles, a
// division 550, so two sums and two quotients cost about 7 us), which two to
// five CTAs per SM overlap.  us per iteration, 2-D grids, CTAs / systems:
//   fp64   1,089 rows x 304: 11.4; 17,424 rows x 14: 13.0 (one CTA per system
//          from L2: 124 for 304 systems); 256 rows x 608: 7.8
//   mixed  1,089 rows x 304: 4.6; 17,424 x 14: 6.6; 256 x 608: 3.5
// Solves: 60 systems of 1,000 - 5,000 rows 8.1 to 3.6 ms (mixed 5.1 to 2.2);
// 300 systems of 200 - 20,000 rows, mixed, 25.5 to 10.4 ms.
#include <algorithm>
#include <climits>

#include "xjpcg_device.cuh"
#include "xjpcg_internal.hpp"

namespace xjpcg {

namespace {
constexpr int kBcMaxCtas = 16;
constexpr int kInfoShared = 1 << 16;  // the slice's rows share their column offsets
constexpr int kInfoLocal = 1 << 17;   // every column of the slice lies in this CTA
constexpr uint64_t kBcWaitNs = 2000000000ull;  // 2 s
constexpr uint32_t kBatchLost = 2;             // status of a system whose CTAs lost one another

// All threads that work on the system.
template <bool MULTI>
__device__ __forceinline__ void system_sync() {
    if (MULTI)
        cluster_sync();
    else
        __syncthreads();
}

__device__ __forceinline__ double bc_load(const double* p, uint32_t rank) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(cluster_addr(p, rank)));
    return v;
}
__device__ __forceinline__ float bc_load(const float* p, uint32_t rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr(p, rank)));
    return v;
}

// This CTA's rows of one system: p and the matrix in shared memory, the matrix
// as 32-row slices (w columns wide, slice-column-major), with 16-bit columns,
// or with the slice's offsets where its rows share them.
template <typename VT>
struct Rows {
    int n, row0, R, ns, w;  // rows of the system; first row, rows and slices of this CTA; slice width
    VT *p, *val;
    uint16_t* col;
    int* info;  // per slice: columns | flags
};

template <typename VT, int NT>
__device__ void load_rows(const Rows<VT>& s, const int* __restrict__ rowptr, const int* __restrict__ col,
                          const double* __restrict__ val) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int ls = wid; ls < s.ns; ls += NT / 32) {
        const int first = s.row0 + 32 * ls, row = first + lane;
        const bool in = row < s.n;
        const int j0 = in ? rowptr[row] : 0, j1 = in ? rowptr[row + 1] : 0;
        VT* const v = s.val + (size_t)ls * 32 * s.w;
        uint16_t* const c = s.col + (size_t)ls * 32 * s.w;
        // the union of the rows' offsets, ascending (as the SELL-32 copy of
        // batched_kernels.cu builds it), when it is no wider than the slices
        bool ok = __all_sync(0xffffffffu, in);
        int L = 0, q = j0, myOff = 0;
        int cur = q < j1 ? col[q] - row : INT_MAX;
        const int most = min(kBatchPatMax, s.w);
        while (ok) {
            const int m = warp_min(cur);
            if (m == INT_MAX) break;
            if (L == most || first + m < 0 || first + 31 + m >= s.n) {
                ok = false;
                break;
            }
            if (lane == L) myOff = m;
            ++L;
            bool bad = false;
            if (cur == m) {
                ++q;
                const int nx = q < j1 ? col[q] - row : INT_MAX;
                bad = nx <= m;
                cur = nx;
            }
            ok = !__any_sync(0xffffffffu, bad);
        }
        if (ok && L > 0) {
            if (lane < L) reinterpret_cast<int*>(c)[lane] = myOff;
            int e = j0;
            for (int k = 0; k < L; ++k) {
                const int o = __shfl_sync(0xffffffffu, myOff, k);
                const bool has = e < j1 && col[e] - row == o;
                v[32 * k + lane] = has ? (VT)val[e] : VT(0);
                if (has) ++e;
            }
            const int lo = __shfl_sync(0xffffffffu, myOff, 0), hi = __shfl_sync(0xffffffffu, myOff, L - 1);
            const bool local = first + lo >= s.row0 && first + 31 + hi < s.row0 + s.R;
            if (lane == 0) s.info[ls] = L | kInfoShared | (local ? kInfoLocal : 0);
        } else {
            const int w = warp_max(j1 - j0);
            bool local = true;
            for (int k = 0; k < w; ++k) {
                const bool has = j0 + k < j1;
                const int cc = has ? col[j0 + k] : (in ? row : s.row0);
                v[32 * k + lane] = has ? (VT)val[j0 + k] : VT(0);
                c[32 * k + lane] = (uint16_t)cc;
                local = local && cc >= s.row0 && cc < s.row0 + s.R;
            }
            local = __all_sync(0xffffffffu, local);
            if (lane == 0) s.info[ls] = w | (local ? kInfoLocal : 0);
        }
    }
}

// p of a column anywhere in the system.
template <typename VT, bool MULTI>
__device__ __forceinline__ VT fetch(const Rows<VT>& s, int c) {
    const int l = c - s.row0;
    if (!MULTI || (unsigned)l < (unsigned)s.R) return s.p[l];
    const int rank = c / s.R;
    return bc_load(s.p + (c - rank * s.R), (uint32_t)rank);
}

template <typename VT, bool MULTI>
__device__ __forceinline__ VT row_dot(const Rows<VT>& s, int ls, int lane) {
    const int info = s.info[ls], w = info & 0xffff;
    const VT* v = s.val + (size_t)ls * 32 * s.w + lane;
    const uint16_t* c = s.col + (size_t)ls * 32 * s.w;
    VT acc = VT(0);
    if (info & kInfoShared) {
        const int* o = reinterpret_cast<const int*>(c);
        const int lr = 32 * ls + lane;
        VT x[kBatchPatMax];
        if (!MULTI || (info & kInfoLocal)) {
            const VT* px = s.p + lr;
#pragma unroll
            for (int u = 0; u < kBatchPatMax; ++u)
                if (u < w) x[u] = px[o[u]];
        } else {
#pragma unroll
            for (int u = 0; u < kBatchPatMax; ++u)
                if (u < w) x[u] = fetch<VT, MULTI>(s, s.row0 + lr + o[u]);
        }
#pragma unroll
        for (int u = 0; u < kBatchPatMax; ++u)
            if (u < w) acc = fma(v[32 * u], x[u], acc);
        return acc;
    }
    c += lane;
    for (int j = 0; j < w; j += 4) {
        VT x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j + u < w) x[u] = fetch<VT, MULTI>(s, (int)c[32 * (j + u)]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j + u < w) acc = fma(v[32 * (j + u)], x[u], acc);
    }
    return acc;
}

// Sums of NV values per thread over the system, the CTAs' parts meeting in
// every CTA's slots: a store that counts itself at the receiver's mbarrier, so
// that no barrier of the cluster and no flush of other stores is in the way.
// slots and bar belong to one kind of sum; two sums of a kind are a barrier of
// the cluster apart.
template <int NT, typename T, int NV>
struct SumBox {
    T part[NV][NT];
    T slots[NV][kBcMaxCtas];
    uint64_t bar;
};

template <typename T>
__device__ __forceinline__ void post(T* slot, uint64_t* bar, uint32_t rank, T v) {
    if constexpr (sizeof(T) == 8)
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(cluster_addr(slot, rank)),
                     "l"(__double_as_longlong(v)), "r"(cluster_addr(bar, rank))
                     : "memory");
    else
        asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(cluster_addr(slot, rank)),
                     "r"(__float_as_uint(v)), "r"(cluster_addr(bar, rank))
                     : "memory");
}

__device__ __forceinline__ bool wait_posts(uint64_t* bar, uint32_t parity) {
    uint64_t t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((spin & 255u) == 255u) {
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > kBcWaitNs) return false;
        }
    }
}

// A wait that gives up.  Shared memory of a CTA that has left may be neither
// written nor read, so no CTA leaves by itself: the one whose wait ran out marks
// all CTAs of the cluster with the number of the cluster's next barrier and goes
// on, with a sum that means nothing, so that the others get its posts.  After
// every barrier of the cluster all compare the mark with that barrier's number
// and leave together, whichever place in the code each came to it from.  The
// missing post may still be on its way: before it leaves, the marking CTA waits
// for it once more.
struct Lost {
    uint32_t mark, parity;
    uint64_t* late;
};

// Threads 0 .. 32 NV - 1 return with the sum of value (their warp) in every
// lane, the others with nothing; the caller syncs the CTA.  Narrow: one warp
// adds all threads' parts of a value (an FP64 add of a warp holds the pipe for
// 16 cycles, whoever needs it).  next: the number of the cluster's next barrier,
// counted from 1.  mute: the CTA's post to the first one stays out (a test of the
// wait's limit).
template <int NT, typename T, int NV, bool MULTI>
__device__ __forceinline__ T system_sum(const T (&v)[NV], SumBox<NT, T, NV>& box, int q, int C, uint32_t parity,
                                        Lost& lost, uint32_t next, bool mute = false) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
#pragma unroll
    for (int i = 0; i < NV; ++i) box.part[i][tid] = v[i];
    if (MULTI && tid == 0) mbar_arrive_expect_tx(&box.bar, (uint32_t)(C * NV * sizeof(T)));
    __syncthreads();
    T t = T(0);
    if (wid < NV) {
        t = box.part[wid][lane];
#pragma unroll
        for (int k = 1; k < NT / 32; ++k) t += box.part[wid][lane + 32 * k];
        t = warp_sum(t);
        if (MULTI) {
            if (lane < C && !(mute && lane == 0)) post(&box.slots[wid][q], &box.bar, (uint32_t)lane, t);
            if (!wait_posts(&box.bar, parity)) {
                lost.parity = parity;
                lost.late = &box.bar;
                if (lane < C)
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr(&lost.mark, (uint32_t)lane)), "r"(next)
                                 : "memory");
            }
            t = warp_sum(lane < C ? box.slots[wid][lane] : T(0));
        }
    }
    return t;
}

// The end of a system whose CTAs lost one another.
__device__ __forceinline__ void end_lost(Lost& lost, BatchResult& res, int q) {
    if (threadIdx.x != 0) return;
    if (q == 0) res.status = kBatchLost;
    if (lost.late != nullptr) wait_posts(lost.late, lost.parity);
}

template <typename VT>
__device__ __forceinline__ Rows<VT> rows_of(const BatchClusterArgs& a, int sys, int q, int C, unsigned char* smem) {
    Rows<VT> s;
    const int r0 = a.sysRow[sys];
    s.n = a.sysRow[sys + 1] - r0;
    s.w = a.width[sys];
    s.R = 32 * (((s.n + 31) / 32 + C - 1) / C);
    s.row0 = q * s.R;
    s.ns = (max(0, min(s.R, s.n - s.row0)) + 31) / 32;
    s.p = reinterpret_cast<VT*>(smem);
    s.val = s.p + s.R;
    s.col = reinterpret_cast<uint16_t*>(s.val + (size_t)s.R * s.w);
    s.info = reinterpret_cast<int*>(s.col + (size_t)s.R * s.w);
    return s;
}
}  // namespace

// FP64.  Thread t owns rows t, t + NT, ... of the CTA in both the product and
// the updates, so r, x, J, z and Ap live in its registers (K rows).
template <int NT, int K, bool MULTI>
__global__ void __launch_bounds__(NT, NT > 256 ? 2 : 5) batch_cluster_fp64_kernel(BatchClusterArgs a) {
    extern __shared__ __align__(16) unsigned char bcSmem[];
    __shared__ SumBox<NT, double, 1> boxA;
    __shared__ SumBox<NT, double, 2> boxB;
    __shared__ double sAlpha, sBeta, sRz, sRr;
    __shared__ int sGo[3];
    __shared__ Lost lost;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int C = MULTI ? a.ctas : 1, q = MULTI ? (int)(blockIdx.x % (unsigned)C) : 0;
    const int sys = a.order[MULTI ? blockIdx.x / (unsigned)C : blockIdx.x];
    const int r0 = a.sysRow[sys];
    const Rows<double> s = rows_of<double>(a, sys, q, C, bcSmem);
    const int rows = max(0, min(s.R, s.n - s.row0));
    if (MULTI) {
        if (tid == 0) {
            lost.mark = 0;
            lost.late = nullptr;
            mbar_init(&boxA.bar, 1);
            mbar_init(&boxB.bar, 1);
            mbar_fence_init();
        }
        cluster_sync();
    }
    // r = b, J = 1 / diag, p = J r, x = 0 (cgVector.hpp:101-114)
    double r[K], x[K], J[K], p[K], z[K];
    double w2[2] = {0.0, 0.0};
#pragma unroll
    for (int u = 0; u < K; ++u) {
        const int i = tid + u * NT;
        r[u] = x[u] = J[u] = p[u] = z[u] = 0.0;
        if (i < rows) {
            r[u] = a.b[r0 + s.row0 + i];
            J[u] = 1.0 / a.diag[r0 + s.row0 + i];
            p[u] = J[u] * r[u];
            s.p[i] = p[u];
            w2[0] = fma(r[u], r[u], w2[0]);
            w2[1] = fma(r[u], p[u], w2[1]);
        }
    }
    load_rows<double, NT>(s, a.rowptr + r0, a.col, a.val);
    {
        const double t = system_sum<NT, double, 2, MULTI>(w2, boxB, q, C, 0u, lost, 1u);
        if (tid == 0) sRr = t;
        if (tid == 32) sRz = t;
    }
    __syncthreads();
    const double rr0 = sRr;
    const double tols = rr0 * a.tol * a.tol;
    system_sync<MULTI>();
    uint32_t k = 0;
    bool go = !MULTI || lost.mark != 1u;
    while (go) {
        // Ap = A p, p.Ap
        double pAp[1] = {0.0};
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (wid + u * (NT / 32) < s.ns) z[u] = row_dot<double, MULTI>(s, wid + u * (NT / 32), lane);
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (tid + u * NT < rows) pAp[0] = fma(p[u], z[u], pAp[0]);
        const double pApT = system_sum<NT, double, 1, MULTI>(pAp, boxA, q, C, k & 1u, lost, k + 2u,
                                                              MULTI && k == a.muteAt && q == C - 1);
        if (tid == 0) {
            const double al = sRz / pApT;
            sAlpha = al;
            sGo[0] = isfinite(al) ? 1 : 0;
        }
        __syncthreads();
        const double alpha = sAlpha;
        w2[0] = w2[1] = 0.0;
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (tid + u * NT < rows) {
                r[u] = fma(-alpha, z[u], r[u]);
                z[u] = r[u] * J[u];
                w2[0] = fma(r[u], r[u], w2[0]);
                w2[1] = fma(r[u], z[u], w2[1]);
            }
        const double tB = system_sum<NT, double, 2, MULTI>(w2, boxB, q, C, (k + 1u) & 1u, lost, k + 2u);
        if (tid == 0) {
            sRr = tB;
            sGo[1] = isfinite(tB) ? (tB >= tols && k + 1u < a.maxIterP1 ? 1 : 0) : 2;
        }
        if (tid == 32) {
            const double beta = tB / sRz;
            sBeta = beta;
            sRz = tB;
            sGo[2] = isfinite(beta) ? 1 : 0;
        }
        // x += alpha p while the first warps collect the sums
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (tid + u * NT < rows) x[u] = fma(alpha, p[u], x[u]);
        __syncthreads();
        const bool broken = sGo[0] == 0 || sGo[1] == 2 || sGo[2] == 0;
        go = !broken && sGo[1] == 1;
        const double beta = sBeta;
        ++k;
        if (go) {
#pragma unroll
            for (int u = 0; u < K; ++u)
                if (tid + u * NT < rows) {
                    p[u] = fma(beta, p[u], z[u]);
                    s.p[tid + u * NT] = p[u];
                }
        } else if (q == 0 && tid == 0) {
            BatchResult& o = a.res[sys];
            o.itersRun = k;
            o.iters = k < a.maxIterP1 ? k : a.maxIterP1 - 1u;
            o.outer = 0;
            o.res = sqrt(sRr / rr0);
            o.status = broken ? 1u : 0u;
        }
        system_sync<MULTI>();
        if (MULTI && lost.mark == k + 1u) break;
    }
    if (MULTI && lost.mark == k + 1u) {
        end_lost(lost, a.res[sys], q);
        return;
    }
#pragma unroll
    for (int u = 0; u < K; ++u)
        if (tid + u * NT < rows) a.x[r0 + s.row0 + tid + u * NT] = x[u];
}

// Mixed precision (reliable updates, as batched_mixed_kernel): FP32 r, d, J, z
// and p, x in global memory, the refresh over the CSR matrix in FP64.
template <int NT, int K, bool MULTI>
__global__ void __launch_bounds__(NT, NT > 128 ? 3 : 6) batch_cluster_mixed_kernel(BatchClusterArgs a) {
    extern __shared__ __align__(16) unsigned char bcSmem[];
    __shared__ SumBox<NT, double, 2> boxR;
    __shared__ SumBox<NT, float, 1> boxA;
    __shared__ SumBox<NT, float, 2> boxB;
    __shared__ double sQ, sT[2];
    __shared__ float sF[2];
    __shared__ Lost lost;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int C = MULTI ? a.ctas : 1, q = MULTI ? (int)(blockIdx.x % (unsigned)C) : 0;
    const int sys = a.order[MULTI ? blockIdx.x / (unsigned)C : blockIdx.x];
    const int r0 = a.sysRow[sys];
    const Rows<float> s = rows_of<float>(a, sys, q, C, bcSmem);
    const int rows = max(0, min(s.R, s.n - s.row0));
    if (MULTI) {
        if (tid == 0) {
            lost.mark = 0;
            lost.late = nullptr;
            mbar_init(&boxR.bar, 1);
            mbar_init(&boxA.bar, 1);
            mbar_init(&boxB.bar, 1);
            mbar_fence_init();
        }
        cluster_sync();
    }
    double* const xs = a.x + r0;  // the system's x
    double* const x = xs + s.row0;
    const double* const b = a.b + r0 + s.row0;
    const int* const rp = a.rowptr + r0;
    // x = 0, d = 0, J = 1/diag, r = b, p = J r
    float r[K], d[K], J[K], p[K], z[K];
    double v2[2] = {0.0, 0.0};
    float rzA = 0.f;
#pragma unroll
    for (int u = 0; u < K; ++u) {
        const int i = tid + u * NT;
        r[u] = d[u] = J[u] = p[u] = z[u] = 0.f;
        if (i < rows) {
            const double bi = b[i];
            J[u] = (float)(1.0 / a.diag[r0 + s.row0 + i]);
            r[u] = (float)bi;
            p[u] = J[u] * r[u];
            s.p[i] = p[u];
            x[i] = 0.0;
            v2[0] = fma(bi, bi, v2[0]);
            rzA = fmaf(r[u], p[u], rzA);
        }
    }
    v2[1] = (double)rzA;
    load_rows<float, NT>(s, rp, a.col, a.val);
    {
        const double t = system_sum<NT, double, 2, MULTI>(v2, boxR, q, C, 0u, lost, 1u);
        if (tid == 0) sT[0] = t;
        if (tid == 32) sT[1] = t;
    }
    __syncthreads();
    const double bb = sT[0];
    double rz = sT[1];
    const double tols = bb * a.tol * a.tol;
    double rrMax = bb, rrTrue = bb;
    uint32_t k = 0, outer = 0;
    bool bd = false, stopped = false;
    system_sync<MULTI>();
    // barriers of the cluster so far: one here, one per iteration and one per refresh
    while (!MULTI || lost.mark != k + outer + 1u) {
        // Ap = A p (FP32), p.Ap
        float pAp[1] = {0.f};
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (wid + u * (NT / 32) < s.ns) z[u] = row_dot<float, MULTI>(s, wid + u * (NT / 32), lane);
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (tid + u * NT < rows) pAp[0] = fmaf(p[u], z[u], pAp[0]);
        const float pApT = system_sum<NT, float, 1, MULTI>(pAp, boxA, q, C, k & 1u, lost, k + outer + 2u,
                                                            MULTI && k == a.muteAt && q == C - 1);
        if (tid == 0) sQ = rz / (double)pApT;
        __syncthreads();
        const double alphaD = sQ;
        const float alpha = (float)alphaD;
        float w2[2] = {0.f, 0.f};
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (tid + u * NT < rows) {
                r[u] = fmaf(-alpha, z[u], r[u]);
                z[u] = r[u] * J[u];
                d[u] = fmaf(alpha, p[u], d[u]);
                w2[0] = fmaf(r[u], r[u], w2[0]);
                w2[1] = fmaf(r[u], z[u], w2[1]);
            }
        const float tB = system_sum<NT, float, 2, MULTI>(w2, boxB, q, C, k & 1u, lost, k + outer + 2u);
        if (tid == 0) sF[0] = tB;
        if (tid == 32) {
            sF[1] = tB;
            sQ = (double)tB / rz;  // beta, unless a refresh is due
        }
        __syncthreads();
        ++k;
        const double rrN = sF[0], rzN = sF[1];
        if (rrN > rrMax) rrMax = rrN;
        bd = !isfinite(alphaD) || !isfinite(rrN) || !isfinite(rzN);
        const bool refresh = bd || rrN < a.delta2 * rrMax || rrN < tols || k + 1u >= a.maxIterP1;
        if (!refresh) {
            rz = rzN;
        } else {
            // fold, FP64 true residual from the CSR matrix, FP32 restart from it
#pragma unroll
            for (int u = 0; u < K; ++u)
                if (tid + u * NT < rows) {
                    x[tid + u * NT] += (double)d[u];
                    d[u] = 0.f;
                }
            system_sync<MULTI>();
            if (MULTI && lost.mark == k + outer + 1u) break;
            double v3[2] = {0.0, 0.0};
            float rzR = 0.f;
#pragma unroll
            for (int u = 0; u < K; ++u) {
                const int i = tid + u * NT;
                if (i < rows) {
                    const int e0 = rp[s.row0 + i], e1 = rp[s.row0 + i + 1];
                    double acc = 0.0;
                    for (int e = e0; e < e1; ++e) acc = fma(a.val[e], xs[a.col[e]], acc);
                    const double ri = b[i] - acc;
                    r[u] = (float)ri;
                    z[u] = r[u] * J[u];
                    v3[0] = fma(ri, ri, v3[0]);
                    rzR = fmaf(r[u], z[u], rzR);
                }
            }
            v3[1] = (double)rzR;
            ++outer;
            const double t = system_sum<NT, double, 2, MULTI>(v3, boxR, q, C, outer & 1u, lost, k + outer + 1u);
            if (tid == 0) sT[0] = t;
            if (tid == 32) {
                sT[1] = t;
                sQ = t / rz;
            }
            __syncthreads();
            rrTrue = sT[0];
            rrMax = rrTrue;
            bool stop = !(rrTrue > tols) || k + 1u >= a.maxIterP1;
            if (bd || !isfinite(rrTrue) || !isfinite(sT[1])) {
                bd = true;
                stop = true;
            }
            rz = sT[1];
            if (stop) {
                stopped = true;
                break;
            }
        }
        const float beta = (float)sQ;
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (tid + u * NT < rows) {
                p[u] = fmaf(beta, p[u], z[u]);
                s.p[tid + u * NT] = p[u];
            }
        system_sync<MULTI>();
    }
    if (stopped) {
        if (q == 0 && tid == 0) {
            BatchResult& o = a.res[sys];
            o.itersRun = k;
            o.iters = k;
            o.outer = outer;
            o.res = sqrt(rrTrue / bb);
            o.status = bd ? 1u : 0u;
        }
        system_sync<MULTI>();  // no CTA leaves while a post to it may be on its way
    }
    if (MULTI && lost.mark == k + outer + 1u) end_lost(lost, a.res[sys], q);
}

// ---------------------------------------------------------------------------
// Checks on the device: flag bits 1 row pointers do not start at 0, 2 row
// pointers are not monotone (then no column is read).
__global__ void batch_rows_kernel(int nsys, int total, const int* __restrict__ sysRow,
                                  const int* __restrict__ rowptr, int* __restrict__ entry, int* flag) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0 && rowptr[0] != 0) atomicOr(flag, 1);
    for (int s = i; s <= nsys; s += gridDim.x * blockDim.x) entry[s] = rowptr[sysRow[s]];
    for (int r = i; r < total; r += gridDim.x * blockDim.x)
        if (rowptr[r + 1] < rowptr[r]) atomicOr(flag, 2);
}

// One thread per row: the longest row of every system, how far its columns reach
// from the diagonal, and flag bit 4 for a column outside its system.
__global__ void batch_widths_kernel(int nsys, int total, const int* __restrict__ sysRow,
                                    const int* __restrict__ rowptr, const int* __restrict__ col, int* __restrict__ width,
                                    int* __restrict__ reach, int* flag) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < total; r += gridDim.x * blockDim.x) {
        int lo = 0, hi = nsys - 1;  // the system of row r
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (sysRow[mid] <= r)
                lo = mid;
            else
                hi = mid - 1;
        }
        const int n = sysRow[lo + 1] - sysRow[lo];
        const int e0 = rowptr[r], e1 = rowptr[r + 1];
        const int row = r - sysRow[lo];
        int far = 0;
        bool bad = false;
        for (int e = e0; e < e1; ++e) {
            const int c = col[e];
            bad = bad || (unsigned)c >= (unsigned)n;
            far = max(far, bad ? 0 : abs(c - row));
        }
        if (bad) atomicOr(flag, 4);
        // most rows are as long as the longest: look before the atomic
        if (*(volatile int*)&width[lo] < e1 - e0) atomicMax(&width[lo], e1 - e0);
        if (*(volatile int*)&reach[lo] < far) atomicMax(&reach[lo], far);
    }
}

cudaError_t batch_check_rows(cudaStream_t st, int nsys, int total, const int* sysRow, const int* rowptr, int* entry,
                             int* flag) {
    batch_rows_kernel<<<std::max(1, std::min((total + 255) / 256, device_sm_count() * 8)), 256, 0, st>>>(
        nsys, total, sysRow, rowptr, entry, flag);
    return cudaGetLastError();
}

cudaError_t batch_widths(cudaStream_t st, int nsys, int total, const int* sysRow, const int* rowptr, const int* col,
                         int* width, int* reach, int* flag) {
    batch_widths_kernel<<<std::max(1, std::min((total + 255) / 256, device_sm_count() * 8)), 256, 0, st>>>(
        nsys, total, sysRow, rowptr, col, width, reach, flag);
    return cudaGetLastError();
}

namespace {
// Threads and rows per thread (in registers) of the small and wide CTAs.
constexpr int kWide64 = 448, kWideRows64 = 3, kWide32 = 256, kWideRows32 = 5;
constexpr int kSmall = 128, kSmallRows = 4;
constexpr size_t kWideSmem = 96 * 1024, kSmallSmem = 40 * 1024;
}  // namespace

int batch_cluster_threads(bool mixed, bool small) { return small ? kSmall : (mixed ? kWide32 : kWide64); }

int batch_cluster_rows(bool mixed, bool small) {
    return small ? kSmall * kSmallRows : (mixed ? kWide32 * kWideRows32 : kWide64 * kWideRows64);
}

size_t batch_cluster_room(bool mixed, bool small) {
    return small ? kSmallSmem : (mixed ? kWideSmem * 2 / 3 : kWideSmem);
}

size_t batch_cluster_smem(bool mixed, int n, int width, int ctas) {
    const size_t ns = ((size_t)(n + 31) / 32 + ctas - 1) / ctas, R = 32 * ns;
    const size_t vt = mixed ? 4 : 8;
    return (R * (vt * (1 + (size_t)width) + 2 * (size_t)width) + 4 * ns + 15) / 16 * 16;
}

namespace {
typedef void (*ClusterKernel)(BatchClusterArgs);

ClusterKernel cluster_kernel(bool mixed, bool small, bool one) {
    if (small)
        return mixed ? (one ? (ClusterKernel)batch_cluster_mixed_kernel<kSmall, kSmallRows, false>
                            : (ClusterKernel)batch_cluster_mixed_kernel<kSmall, kSmallRows, true>)
                     : (one ? (ClusterKernel)batch_cluster_fp64_kernel<kSmall, kSmallRows, false>
                            : (ClusterKernel)batch_cluster_fp64_kernel<kSmall, kSmallRows, true>);
    return mixed ? (one ? (ClusterKernel)batch_cluster_mixed_kernel<kWide32, kWideRows32, false>
                        : (ClusterKernel)batch_cluster_mixed_kernel<kWide32, kWideRows32, true>)
                 : (one ? (ClusterKernel)batch_cluster_fp64_kernel<kWide64, kWideRows64, false>
                        : (ClusterKernel)batch_cluster_fp64_kernel<kWide64, kWideRows64, true>);
}

cudaError_t cluster_config(ClusterKernel k, bool mixed, bool small, int systems, int ctas, size_t smem,
                           cudaStream_t st, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmem);
    if (e == cudaSuccess && ctas > 8) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    *cfg = {};
    cfg->gridDim = dim3((unsigned)(systems * ctas));
    cfg->blockDim = dim3((unsigned)batch_cluster_threads(mixed, small));
    cfg->dynamicSmemBytes = smem;
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = ctas > 1 ? 1 : 0;
    return e;
}
}  // namespace

// Asked once per device, kernel and size.
bool batch_cluster_offered(bool mixed, bool small, int ctas) {
    if (ctas == 1) return true;
    constexpr int kMaxDev = 64;
    static int cache[kMaxDev][2][2][kBcMaxCtas + 1] = {};  // 0 not asked, 1 yes, 2 no
    int dev = 0;
    if (ctas > kBcMaxCtas || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) {
        cudaGetLastError();
        return false;
    }
    int* const known = &cache[dev][mixed][small][ctas];
    int v = __atomic_load_n(known, __ATOMIC_RELAXED);
    if (v == 0) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        const ClusterKernel k = cluster_kernel(mixed, small, false);
        int clusters = 0;
        v = cluster_config(k, mixed, small, 1, ctas, batch_cluster_room(mixed, small), nullptr, &cfg, attr) ==
                        cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) == cudaSuccess && clusters > 0
                ? 1
                : 2;
        cudaGetLastError();
        __atomic_store_n(known, v, __ATOMIC_RELAXED);
    }
    return v == 1;
}

cudaError_t batch_cluster_launch(cudaStream_t st, bool mixed, bool small, int systems, size_t smem,
                                 const BatchClusterArgs& a) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const ClusterKernel k = cluster_kernel(mixed, small, a.ctas == 1);
    const cudaError_t e = cluster_config(k, mixed, small, systems, a.ctas, smem, st, &cfg, attr);
    return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, k, a) : e;
}

}  // namespace xjpcg
