// cg_loop.cu -- the whole fp64 JPCG loop in one kernel, for systems whose
// vectors fit on the chip.
//
// What bounds a small system is the chain of dependent steps in an iteration,
// not bytes or operations: on GB300 a dependent FP64 add takes 64 cycles, a
// division 550, a load from L2 300 and more, a release fence 540, a counter
// barrier over 152 SMs 1,600 and a cluster barrier 370 (all measured).  As two
// kernels per iteration in a graph, with a grid barrier inside the second, an
// iteration took 14 to 15 us however small the system.  Here one launch runs
// all iterations, and r, x, z = J r, p and (if it fits) J never leave shared
// memory; p is also written to global memory, for the other CTAs' gathers.
//
// Two forms:
//   cg_cluster_kernel  one cluster of up to 16 CTAs; p is gathered, and the
//                      sums are exchanged, through distributed shared memory;
//                      the matrix stays on the chip.  Three cluster barriers
//                      per iteration.
//   cg_loop_kernel     one CTA per SM, cooperative; sums go through posts and
//                      counters in global memory, the matrix streams from L2.
//
// A larger system is bound by FP64 issue (14 operations per row and iteration
// with 7 entries in a row, 34 with 27; 2 per clock and SM) as long as loads and
// the 64-cycle FMAs of a row overlap.  With 12 warps per SM they do so only when
// each warp works on three steps at once: columns of one on their way, values
// and p of the next, sums of the one before, instruction by instruction.  7-point
// 96^3 32.4 us per iteration: 27,700 cycles for the product (23,300 of issue at
// the least), 14,700 for r and z, 5,000 for p, the rest waiting for sums.
// Loading values and columns a step ahead but gathering when needed took 48.7
// us, the three stages one after another 39.2.  Keeping the matrix in what is
// left of shared memory gained nothing over streaming it (7-point 32^3 9.5 us
// either way, 64^3 16.9 and 16.8; 27-point 48^3 17.9 and 17.4).
//
// Measured, us per iteration (two kernels per iteration / loop / cluster):
//   7-point   16^3   14.7 /  8.8 / 5.7      27-point   8^3  15.1 / 13.1 / 6.3
//             24^3   15.1 /  8.9 / 8.5                16^3  16.9 / 10.2 / 7.6
//             32^3   14.9 /  9.5 /  -                 32^3  18.6 / 11.2 /  -
//             48^3   18.1 / 11.4 /  -                 48^3  24.6 / 16.8 /  -
//             64^3   25.1 / 15.9 /  -                 60^3  32.7 / 23.1 /  -
//             80^3   33.1 / 22.1 /  -                 80^3  50.3 / 40.2 /  -
//             96^3   42.2 / 32.4 /  -                 96^3  73.5 / 61.9 /  -
//            102^3   44.9 / 37.2 /  -                102^3  81.7 / 72.1 /  -
// (sums by a shuffle tree in every warp: cluster 16^3 6.6, 20^3 9.0 against 7.2)
//
// Every row is summed in its stored order, as in the sliced SpMV kernels; the
// dot products are summed per thread, per warp, per CTA and over the CTAs, in
// an order that depends on n and the entries stored, not on the layout, so a solve
// is bitwise reproducible.
#include <algorithm>

#include "xjpcg_device.cuh"
#include "xjpcg_internal.hpp"

namespace xjpcg {

namespace {
constexpr int kLoopThreads = 384;   // 168 registers; with 512 (128 registers) the pipelined steps spill
constexpr int kVecThreads = 256;    // threads that update r and z: enough to fill the FP64 pipe, and every warp costs two sums
constexpr int kStep[2] = {7, 9};    // stored columns per step of a row
constexpr int kCols = 8;            // the same in the cluster form
constexpr int kPosts = 5;           // posts a lane reads at once: 152 CTAs in one step
constexpr uint64_t kLoopBudgetNs = 2000000000ull;  // 2 s
constexpr size_t kLoopSmem = 226 * 1024;

__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// Waits until the counter has reached target.  False after the wait's budget.
// One thread per CTA polls one address: 152 CTAs meet in 1,600 cycles, where
// every CTA polling every CTA's flag took 8,900 (the few lines that all read).
__device__ __forceinline__ bool wait_count(const uint32_t* counter, uint32_t target) {
    uint64_t t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        uint32_t v;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
        if ((int32_t)(v - target) >= 0) return true;
        if ((spin & 255u) == 255u) {
            const uint64_t now = globaltimer_ns();
            if (t0 == 0) t0 = now;
            if (now - t0 > kLoopBudgetNs) return false;
        }
    }
}

__device__ __forceinline__ void arrive(uint32_t* counter) {
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
}

// Sum over the lanes below `count` (a power of two or 32), in lane 0 at least.
// A dependent FP64 add takes 64 cycles here, so no level is taken in vain.
__device__ __forceinline__ double lanes_sum(double v, int count) {
    for (int o = 16; o > 0; o >>= 1)
        if (o < count) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// This thread's warp, as a value that the compiler knows to be the same in all
// lanes: shuffles under a test of it need no reconvergence.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }

// Sum of the values that nw warps' threads left in shared memory, by one warp:
// over the lanes in groups of `width`, in each group's first lane.  A warp-wide add
// holds the SM's FP64 pipe for 16 cycles: a shuffle tree in each of 8 warps is 40
// of them, this is 12 for all.
__device__ __forceinline__ double threads_sum(const double* v, int nw, int lane, int width = 32) {
    double s[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = u < nw ? v[u * 32 + lane] : 0.0;
    for (int w = 4; w < nw; w += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (w + u < nw) s[u] += v[(w + u) * 32 + lane];
    return lanes_sum((s[0] + s[1]) + (s[2] + s[3]), width);
}

// A CTA's total to every CTA and back, by one warp: the sum of all CTAs'
// totals, in every lane.  A post is two words of half the value and the
// iteration's tag, so it needs no fence before the counter: the counter says
// when to look, the tags say whether the post has landed.
__device__ __forceinline__ double grid_total(double s, ulonglong2* posts, uint32_t* counter, uint32_t target,
                                             uint32_t tag, int lane, bool& ok) {
    if (lane == 0) {
        const uint64_t bits = (uint64_t)__double_as_longlong(s);
        const uint64_t lo = (bits & 0xffffffffull) | ((uint64_t)tag << 32), hi = (bits >> 32) | ((uint64_t)tag << 32);
        asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(posts + blockIdx.x), "l"(lo), "l"(hi)
                     : "memory");
        arrive(counter);
        ok = wait_count(counter, target);
    }
    __syncwarp();
    double sum = 0.0;
    uint64_t t0 = 0;
    const int P = gridDim.x;
    for (int b = lane; b < P; b += 32 * kPosts) {
        ulonglong2 w[kPosts];
        for (uint32_t spin = 0;; ++spin) {
            bool all = true;
#pragma unroll
            for (int u = 0; u < kPosts; ++u)
                if (b + 32 * u < P)
                    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];"
                                 : "=l"(w[u].x), "=l"(w[u].y)
                                 : "l"(posts + b + 32 * u)
                                 : "memory");
#pragma unroll
            for (int u = 0; u < kPosts; ++u)
                if (b + 32 * u < P) all = all && (uint32_t)(w[u].x >> 32) == tag && (uint32_t)(w[u].y >> 32) == tag;
            if (all) break;
            if ((spin & 255u) == 255u) {
                const uint64_t now = globaltimer_ns();
                if (t0 == 0) t0 = now;
                if (now - t0 > kLoopBudgetNs) {
                    ok = false;
                    break;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kPosts; ++u)
            if (b + 32 * u < P)
                sum += __longlong_as_double((long long)((w[u].x & 0xffffffffull) | (w[u].y << 32)));
    }
    __syncwarp();
    return warp_sum(sum);
}
}  // namespace

// One step of a row, up to K stored columns.
template <int K>
struct Step {
    double v[K], x[K];
    int ls, rem;  // slice; its columns from this step's first on
};
// A step's place in the matrix.
struct StepAt {
    int ls, rem;
    int v, c;    // of its values; of its columns
    int shared;  // columns: offsets shared by the slice
};

// CTA q owns a contiguous run of slices (so neighbouring rows' gathers meet in
// its L1).  Per iteration:
//   Ap = A p into sz, p.Ap        -> grid sum, alpha
//   r -= alpha Ap, z = J r        -> grid sums of r.r and r.z, beta, stop test;
//                                    the other warps do x += alpha p meanwhile
//   p = z + beta p, also to global -> barrier (release / acquire)
// Only the last needs fences: the posts of the sums carry their own tags.
// LAY: 0 int32 columns, 1 int16 offsets, 2 slice-shared offsets.
// K: stored columns per step.
template <int LAY, int K>
__global__ void __launch_bounds__(kLoopThreads, 1) cg_loop_kernel(LoopArgs a) {
    extern __shared__ __align__(16) unsigned char loopSmem[];
    __shared__ double sAlpha, sBeta, sRz, sRr;
    __shared__ int sGo[3];
    const int tid = threadIdx.x, lane = tid & 31, wid = warp_index(), nt = blockDim.x, nw = nt >> 5;
    const int q = blockIdx.x, P = gridDim.x;
    const int s0 = (int)((int64_t)a.nslices * q / P), s1 = (int)((int64_t)a.nslices * (q + 1) / P);
    const int ns = s1 - s0, pairs = ns * 16, row0 = s0 * 32;
    double* const sr = reinterpret_cast<double*>(loopSmem);
    double* const sx = sr + a.rows;
    double* const sz = sx + a.rows;
    double* const sp = sz + a.rows;
    double* const sj = sp + a.rows;
    double* const part = sj + (a.jOnChip ? a.rows : 0);  // 1 per thread
    int4* const meta = reinterpret_cast<int4*>(part + kLoopThreads);

    for (int i = tid; i < pairs; i += nt) {
        const int e = row0 / 2 + i;
        const bool in = e < a.n2;
        const double2 zero = make_double2(0.0, 0.0);
        reinterpret_cast<double2*>(sr)[i] = in ? reinterpret_cast<const double2*>(a.r)[e] : zero;
        reinterpret_cast<double2*>(sp)[i] = in ? reinterpret_cast<const double2*>(a.p)[e] : zero;
        if (a.jOnChip) reinterpret_cast<double2*>(sj)[i] = in ? reinterpret_cast<const double2*>(a.J)[e] : zero;
        reinterpret_cast<double2*>(sx)[i] = zero;
    }
    // slice records: {first value, columns, pattern or first column, shared offsets?}
    for (int i = tid; i < ns; i += nt) {
        const int off = a.sliceOff[s0 + i];
        int4 md = make_int4(off, (a.sliceOff[s0 + i + 1] - off) >> 5, off, 0);
        if (LAY == 2) {
            md.w = a.patLen[s0 + i] > 0 ? 1 : 0;
            md.z = md.w ? a.patOff[a.patIdx[s0 + i]] : a.genOff[s0 + i];
        }
        meta[i] = md;
    }
    if (tid == 0) sRz = a.state->rz;
    __syncthreads();
    const double tols = a.state->tols;
    const uint32_t maxIterP1 = a.state->maxIterP1;
    double2* const p2 = reinterpret_cast<double2*>(a.p) + row0 / 2;
    const int have2 = max(0, min(pairs, a.n2 - row0 / 2));  // pairs of this CTA that exist

    // shared or global, read through one pointer
    const double2* const j2 = a.jOnChip ? reinterpret_cast<const double2*>(sj) : reinterpret_cast<const double2*>(a.J) + row0 / 2;
    const int vecStride = min(nt, kVecThreads);

    // A step passes through three stages: its columns are loaded, then its values
    // and p, then the products are summed.  A warp has one step in each.
    int cols[K];
    Step<K> A, B;
    auto slice = [&](int ls) {
        const int4 md = meta[min(ls, ns - 1)];
        StepAt t;
        t.ls = ls;
        t.rem = ls < ns ? md.y : 0;
        t.v = md.x + lane;
        t.shared = LAY == 2 ? md.w : 0;
        t.c = t.shared ? md.z : md.z + lane;
        return t;
    };
    auto next = [&](const StepAt& t) {
        if (t.rem <= K) return slice(t.ls + nw);
        StepAt l = t;
        l.rem -= K;
        l.v += K * 32;
        l.c += t.shared ? K : K * 32;
        return l;
    };
    auto load_col = [&](const StepAt& t, int u) {
        if (LAY == 0) return __ldcs(a.col32 + t.c + u * 32);
        if (LAY == 1) return (int)__ldcs(a.col16 + t.c + u * 32);
        return __ldg((t.shared ? a.pat : a.gcol) + t.c + (t.shared ? u : u * 32));
    };
    auto base_of = [&](const StepAt& t) {
        const int row = row0 + t.ls * 32 + lane;
        return a.p + (LAY == 0 ? 0 : (LAY == 1 ? min(row, a.n - 1) : (t.shared ? row : 0)));
    };
    auto start = [&]() {
        if (wid >= ns) return;
        const StepAt t = slice(wid);
#pragma unroll
        for (int u = 0; u < K; ++u)
            if (u < t.rem) {
                cols[u] = load_col(t, u);
                A.v[u] = ld_val(a.sval + t.v + u * 32);
            }
    };
    start();

    uint32_t k = 0;
    bool ok = true;
    for (;;) {
        const uint32_t target = (k + 1u) * (uint32_t)P, tag = a.tag0 + k;
        // ---- Ap = A p (kept in sz) and this thread's part of p.Ap ----
        double dacc = 0.0;
        if (wid < ns) {
            double acc = 0.0;
            StepAt pos = slice(wid);
            A.ls = wid;
            A.rem = pos.rem;
            {
                const double* const pb = base_of(pos);
                const StepAt l = next(pos);
#pragma unroll
                for (int u = 0; u < K; ++u) {
                    if (u < pos.rem) A.x[u] = pb[cols[u]];
                    if (u < l.rem) cols[u] = load_col(l, u);
                }
                pos = l;
            }
            auto finish = [&](const Step<K>& f) {
                if (f.rem > K) return;  // more of the slice to come
                const int r = f.ls * 32 + lane;
                const bool in = row0 + r < a.n;
                sz[r] = in ? acc : 0.0;
                if (in) dacc = fma(sp[r], acc, dacc);
                acc = 0.0;
            };
            auto step = [&](const Step<K>& f, Step<K>& g) {  // pos: g's place
                if (pos.ls >= ns) {  // f is the warp's last
#pragma unroll
                    for (int u = 0; u < K; ++u)
                        if (u < f.rem) acc = fma(f.v[u], f.x[u], acc);
                    finish(f);
                    return false;
                }
                const StepAt l = next(pos);
                const double* const pb = base_of(pos);
                const double* const vp = a.sval + pos.v;
                g.ls = pos.ls;
                g.rem = pos.rem;
                // the stages' instructions alternate, as a dependent FMA takes 64 cycles
                if (min(min(f.rem, pos.rem), l.rem) >= K) {
#pragma unroll
                    for (int u = 0; u < K; ++u) {
                        g.x[u] = pb[cols[u]];
                        g.v[u] = ld_val(vp + u * 32);
                        cols[u] = load_col(l, u);
                        acc = fma(f.v[u], f.x[u], acc);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < K; ++u) {
                        if (u < pos.rem) {
                            g.x[u] = pb[cols[u]];
                            g.v[u] = ld_val(vp + u * 32);
                        }
                        if (u < l.rem) cols[u] = load_col(l, u);
                        if (u < f.rem) acc = fma(f.v[u], f.x[u], acc);
                    }
                }
                finish(f);
                pos = l;
                return true;
            };
            while (step(A, B) && step(B, A)) {
            }
        }
        part[tid] = dacc;
        __syncthreads();
        if (wid == 0) {
            double s = threads_sum(part, nw, lane);
            s = grid_total(s, a.posts, a.counters, target, tag, lane, ok);
            if (lane == 0) {
                const double al = sRz / s;
                sAlpha = al;
                sGo[0] = isfinite(al) ? 1 : 0;
                if (q == 0) a.state->pAp = s;
            }
        }
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        const double alpha = sAlpha;
        // ---- r -= alpha Ap, z = J r ----
        double rr = 0.0, rz = 0.0;
        double2 jn = make_double2(0.0, 0.0);
        if (tid < min(have2, kVecThreads)) jn = j2[tid];
        for (int i = tid; i < have2 && tid < kVecThreads; i += vecStride) {
            double2 rv = reinterpret_cast<double2*>(sr)[i];
            const double2 av = reinterpret_cast<double2*>(sz)[i], jv = jn;
            if (i + vecStride < have2) jn = j2[i + vecStride];
            rv.x = fma(-alpha, av.x, rv.x);
            rv.y = fma(-alpha, av.y, rv.y);
            const double2 zv = make_double2(rv.x * jv.x, rv.y * jv.y);
            rr = fma(rv.x, rv.x, rr);
            rr = fma(rv.y, rv.y, rr);
            rz = fma(rv.x, zv.x, rz);
            rz = fma(rv.y, zv.y, rz);
            reinterpret_cast<double2*>(sr)[i] = rv;
            reinterpret_cast<double2*>(sz)[i] = zv;
        }
        if (tid < kVecThreads) {
            // the lower lanes go on with r.r, the upper with r.z
            const double other = __shfl_xor_sync(0xffffffffu, lane < 16 ? rz : rr, 16);
            part[tid] = (lane < 16 ? rr : rz) + other;
        }
        __syncthreads();
        auto updateX = [&](int from, int step) {
            for (int i = from; i < have2; i += step) {
                double2 xv = reinterpret_cast<double2*>(sx)[i];
                const double2 pv = reinterpret_cast<double2*>(sp)[i];
                xv.x = fma(alpha, pv.x, xv.x);
                xv.y = fma(alpha, pv.y, xv.y);
                reinterpret_cast<double2*>(sx)[i] = xv;
            }
        };
        if (wid < 2) {
            double s = threads_sum(part, min(nw, kVecThreads / 32), lane, 16);
            s = __shfl_sync(0xffffffffu, s, 16 * wid);
            s = grid_total(s, a.posts + (1 + wid) * P, a.counters + (1 + wid) * 32, target, tag, lane, ok);
            if (lane == 0) {
                if (wid == 0) {
                    sRr = s;
                    sGo[1] = isfinite(s) && !(s < tols) && k + 1u < maxIterP1 ? 1 : 0;
                } else {
                    const double beta = s / sRz;
                    sBeta = beta;
                    sRz = s;
                    sGo[2] = isfinite(beta) ? 1 : 0;
                }
            }
        } else {
            // x += alpha p while the sums are on their way
            updateX(tid - 64, nt - 64);
        }
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        const bool go = (sGo[0] & sGo[1] & sGo[2]) != 0;
        const double beta = sBeta;
        if (q == 0 && tid == nt - 1) {
            CgState* st = a.state;
            write_record(st, k, sRr, sRz, alpha, beta);
            if (!go) {
                st->alpha = alpha;
                st->rr = sRr;
                st->rz = sRz;
                st->beta = beta;
                st->k = k + 1u;
                if (!isfinite(alpha) || !isfinite(beta) || !isfinite(sRr)) st->status |= kStatusBreakdown;
                st->done = 1u;
            }
        }
        if (nt == 64) updateX(tid, nt);  // no third warp
        if (!go) break;
        // ---- p = z + beta p ----
        for (int i = tid; i < have2; i += nt) {
            double2 pv = reinterpret_cast<double2*>(sp)[i];
            const double2 zv = reinterpret_cast<double2*>(sz)[i];
            pv.x = fma(beta, pv.x, zv.x);
            pv.y = fma(beta, pv.y, zv.y);
            reinterpret_cast<double2*>(sp)[i] = pv;
            p2[i] = pv;
        }
        __syncthreads();
        if (tid == 0) {
            fence_gpu();
            arrive(a.counters + 96);
        }
        start();  // after the arrival, which the other CTAs wait for
        if (tid == 0) {
            ok = wait_count(a.counters + 96, target);
            fence_gpu();
        }
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        ++k;
    }
    if (!ok) {
        if (tid == 0) {
            atomicOr(&a.state->status, kStatusWaitTimeout);
            a.state->done = 1u;
        }
        return;
    }
    for (int i = tid; i < have2; i += nt)
        reinterpret_cast<double2*>(a.x)[row0 / 2 + i] = reinterpret_cast<double2*>(sx)[i];
}

namespace {
constexpr int kClusterThreads = 512;
constexpr int kClusterMax = 16;
constexpr size_t kClusterSmem = 212 * 1024;  // beside 14 KB of static shared memory

__device__ __forceinline__ double ld_cluster(uint32_t a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}

// v, in every lane, into the same place of every CTA of the cluster.
__device__ __forceinline__ void to_all(double* place, double v, int P, int lane) {
    if (lane < P)
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(cluster_addr(place, (uint32_t)lane)), "d"(v) : "memory");
}

}  // namespace

// One cluster.  R rows per CTA, so a column's owner is column / R.  The matrix,
// in shared memory, holds per entry the value and the cluster address of its p,
// so a gather is one load (about 250 cycles; 4.5 cycles more per entry and CTA
// where the lanes' addresses lie scattered).  NARROW: 16-bit column offsets.  Every CTA writes its part
// of a sum to every CTA; after the cluster barrier each adds all of them in the
// same order.  A CTA always runs to the same decision as the others, and no
// CTA is read or written by another after its last cluster barrier.
template <bool NARROW>
__global__ void __launch_bounds__(kClusterThreads, 1) cg_cluster_kernel(LoopArgs a) {
    extern __shared__ __align__(16) unsigned char loopSmem[];
    __shared__ double slots[3][kClusterMax], part[2][kClusterThreads];
    __shared__ double sAlpha, sBeta, sRz, sRr;
    __shared__ int sGo[3];
    const int tid = threadIdx.x, lane = tid & 31, wid = warp_index(), nt = blockDim.x, nw = nt >> 5;
    const int q = blockIdx.x, P = gridDim.x, R = a.rows;
    const int s0 = q * (R / 32), ns = max(0, min(R / 32, a.nslices - s0)), row0 = s0 * 32;
    double* const sr = reinterpret_cast<double*>(loopSmem);
    double* const sx = sr + R;
    double* const sz = sx + R;
    double* const sp = sz + R;
    double* const sj = sp + R;
    int2* const meta = reinterpret_cast<int2*>(sj + R);
    double* const mv = reinterpret_cast<double*>(meta + R / 32);
    for (int i = tid; i < R; i += nt) {
        const int e = row0 + i;
        const bool in = e < 2 * a.n2;
        sr[i] = in ? a.r[e] : 0.0;
        sp[i] = in ? a.p[e] : 0.0;
        sj[i] = in ? a.J[e] : 0.0;
        sx[i] = 0.0;
    }
    for (int i = tid; i < ns; i += nt) {  // slice records: {first value, columns}
        const int off = a.sliceOff[s0 + i];
        meta[i] = make_int2(off, (a.sliceOff[s0 + i + 1] - off) >> 5);
    }
    if (tid == 0) sRz = a.state->rz;
    __syncthreads();
    const int mat0 = ns > 0 ? meta[0].x : 0;
    const int matN = ns > 0 ? meta[ns - 1].x + 32 * meta[ns - 1].y - mat0 : 0;
    uint32_t* const mc = reinterpret_cast<uint32_t*>(mv + matN);
    // where an entry's row finds its p, in the cluster's shared memory
    for (int ls = wid; ls < ns; ls += nw) {
        const int2 md = meta[ls];
        const int row = min(row0 + ls * 32 + lane, a.n - 1);
        for (int j = 0; j < md.y; ++j) {
            const int e = md.x + j * 32 + lane, c = NARROW ? row + a.col16[e] : a.col32[e];
            mv[e - mat0] = a.sval[e];
            mc[e - mat0] = cluster_addr(sp + c % R, (uint32_t)(c / R));
        }
    }
    const double tols = a.state->tols;
    const uint32_t maxIterP1 = a.state->maxIterP1;
    cluster_sync();

    uint32_t k = 0;
    bool go = true;
    while (go) {
        // ---- Ap = A p ----
        double dacc = 0.0;
        for (int ls = wid; ls < ns; ls += nw) {
            const int2 md = meta[ls];
            const int r = ls * 32 + lane;
            double acc = 0.0;
            const int at = md.x - mat0 + lane;
            for (int j = 0; j < md.y; j += kCols) {
                double xv[kCols];
#pragma unroll
                for (int u = 0; u < kCols; ++u)
                    if (j + u < md.y) xv[u] = ld_cluster(mc[at + (j + u) * 32]);
#pragma unroll
                for (int u = 0; u < kCols; ++u)
                    if (j + u < md.y) acc = fma(mv[at + (j + u) * 32], xv[u], acc);
            }
            if (row0 + r >= a.n) acc = 0.0;
            sz[r] = acc;
            dacc = fma(sp[r], acc, dacc);
        }
        part[0][tid] = dacc;
        __syncthreads();
        if (wid == 0) to_all(&slots[0][q], threads_sum(part[0], nw, lane), P, lane);
        cluster_sync();
        if (wid == 0) {
            const double s = lanes_sum(lane < P ? slots[0][lane] : 0.0, kClusterMax);
            if (lane == 0) {
                const double al = sRz / s;
                sAlpha = al;
                sGo[0] = isfinite(al) ? 1 : 0;
                if (q == 0) a.state->pAp = s;
            }
        }
        __syncthreads();
        const double alpha = sAlpha;
        // ---- r -= alpha Ap, z = J r ----
        double rr = 0.0, rz = 0.0;
        for (int i = tid; i < ns * 32; i += nt) {
            const double rv = fma(-alpha, sz[i], sr[i]);
            const double zv = rv * sj[i];
            rr = fma(rv, rv, rr);
            rz = fma(rv, zv, rz);
            sr[i] = rv;
            sz[i] = zv;
        }
        part[0][tid] = rr;
        part[1][tid] = rz;
        __syncthreads();
        if (wid < 2) to_all(&slots[1 + wid][q], threads_sum(part[wid], nw, lane), P, lane);
        cluster_sync();
        if (wid < 2) {
            const double s = lanes_sum(lane < P ? slots[1 + wid][lane] : 0.0, kClusterMax);
            if (lane == 0) {
                if (wid == 0) {
                    sRr = s;
                    sGo[1] = isfinite(s) && !(s < tols) && k + 1u < maxIterP1 ? 1 : 0;
                } else {
                    const double beta = s / sRz;
                    sBeta = beta;
                    sRz = s;
                    sGo[2] = isfinite(beta) ? 1 : 0;
                }
            }
        }
        __syncthreads();
        go = (sGo[0] & sGo[1] & sGo[2]) != 0;
        const double beta = sBeta;
        if (q == 0 && tid == nt - 1) {
            CgState* st = a.state;
            write_record(st, k, sRr, sRz, alpha, beta);
            if (!go) {
                st->alpha = alpha;
                st->rr = sRr;
                st->rz = sRz;
                st->beta = beta;
                st->k = k + 1u;
                if (!isfinite(alpha) || !isfinite(beta) || !isfinite(sRr)) st->status |= kStatusBreakdown;
                st->done = 1u;
            }
        }
        // ---- x += alpha p, p = z + beta p ----
        for (int i = tid; i < ns * 32; i += nt) {
            const double pv = sp[i];
            sx[i] = fma(alpha, pv, sx[i]);
            if (go) sp[i] = fma(beta, pv, sz[i]);
        }
        if (go) cluster_sync();
        ++k;
    }
    for (int i = tid; i < ns * 32; i += nt)
        if (row0 + i < 2 * a.n2) a.x[row0 + i] = sx[i];
}

namespace {
struct LoopShape {
    int P, rows, threads;
    bool jOnChip;  // grid form: J in shared memory as well
    size_t fixed;  // shared memory besides the matrix
};

LoopShape loop_shape(int n, int numSms) {
    LoopShape s;
    const int nslices = (n + 31) / 32;
    s.P = std::min(numSms, nslices);
    const int ns = (nslices + s.P - 1) / s.P;
    s.rows = 32 * ns;
    s.threads = std::max(64, std::min(kLoopThreads, 32 * ns));
    const size_t other = sizeof(double) * kLoopThreads + sizeof(int4) * (size_t)ns;
    s.jOnChip = sizeof(double) * 5 * (size_t)s.rows + other <= kLoopSmem;
    s.fixed = sizeof(double) * (s.jOnChip ? 5 : 4) * (size_t)s.rows + other;
    return s;
}

template <int LAY, int K>
cudaError_t loop_launch(cudaStream_t st, const LoopShape& s, const LoopArgs& a) {
    cudaError_t e = cudaFuncSetAttribute(cg_loop_kernel<LAY, K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kLoopSmem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)s.P);
    cfg.blockDim = dim3((unsigned)s.threads);
    cfg.dynamicSmemBytes = s.fixed;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, cg_loop_kernel<LAY, K>, a);
}

template <int LAY>
cudaError_t loop_launch_steps(int step, cudaStream_t st, const LoopShape& s, const LoopArgs& a) {
    return step == kStep[1] ? loop_launch<LAY, kStep[1]>(st, s, a) : loop_launch<LAY, kStep[0]>(st, s, a);
}

// The cluster form: its CTAs' rows and shared memory.
LoopShape cluster_shape(int n) {
    LoopShape s;
    const int nslices = (n + 31) / 32;
    const int ns = (nslices + kClusterMax - 1) / kClusterMax;
    s.P = (nslices + ns - 1) / ns;
    s.rows = 32 * ns;
    s.threads = std::max(64, std::min(kClusterThreads, 32 * ns));
    s.fixed = sizeof(double) * 5 * (size_t)s.rows + sizeof(int2) * (size_t)(ns + ns % 2);
    return s;
}

template <bool NARROW>
cudaError_t cluster_config(const LoopShape& s, size_t smem, cudaStream_t st, cudaLaunchConfig_t* cfg,
                           cudaLaunchAttribute* attr) {
    cudaError_t e = cudaFuncSetAttribute(cg_cluster_kernel<NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)kClusterSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(cg_cluster_kernel<NARROW>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    *cfg = {};
    cfg->gridDim = dim3((unsigned)s.P);
    cfg->blockDim = dim3((unsigned)s.threads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)s.P;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg->attrs = attr;
    cfg->numAttrs = 1;
    return e;
}

// Whether the current device can hold the largest cluster; asked once per device.
bool device_takes_cluster() {
    constexpr int kMaxDev = 64;
    static int cache[kMaxDev] = {};  // 0 not asked, 1 yes, 2 no
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) {
        cudaGetLastError();
        return false;
    }
    int v = __atomic_load_n(&cache[dev], __ATOMIC_RELAXED);
    if (v == 0) {
        LoopShape s;
        s.P = kClusterMax;
        s.threads = kClusterThreads;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute attr[1];
        int clusters = 0;
        v = cluster_config<true>(s, kClusterSmem, nullptr, &cfg, attr) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&clusters, cg_cluster_kernel<true>, &cfg) == cudaSuccess && clusters > 0
                ? 1
                : 2;
        cudaGetLastError();
        __atomic_store_n(&cache[dev], v, __ATOMIC_RELAXED);
    }
    return v == 1;
}

template <bool NARROW>
cudaError_t cluster_launch(cudaStream_t st, const LoopShape& s, const LoopArgs& a) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    const cudaError_t e = cluster_config<NARROW>(s, a.smem, st, &cfg, attr);
    return e == cudaSuccess ? cudaLaunchKernelEx(&cfg, cg_cluster_kernel<NARROW>, a) : e;
}
}  // namespace

// FP64 operations of an iteration up to which 16 SMs finish before 152 do.  us per
// iteration, cluster / grid: 7-point 20^3 (112,000) 7.2 / 9.1, 24^3 (194,000) 8.5 /
// 8.9, 26^3 (246,000) 9.9 / 9.0; 27-point 16^3 (139,000) 7.6 / 10.2, 18^3 (198,000)
// 9.0 / 10.7, 20^3 (272,000) 10.6 / 10.6.
constexpr int64_t kClusterWork = 210000;

bool cg_cluster_fits(int n, int64_t stored, const LoopBalance& b) {
    if (n <= 0 || stored + 7 * (int64_t)n > kClusterWork) return false;
    if (cluster_shape(n).fixed + 32 * 12 * (size_t)b.clusterCols > kClusterSmem) return false;
    return device_takes_cluster();
}

cudaError_t cg_cluster_launch(cudaStream_t st, bool narrow, LoopArgs a) {
    const LoopShape s = cluster_shape(a.n);
    a.nslices = (a.n + 31) / 32;
    a.rows = s.rows;
    a.smem = kClusterSmem;  // whatever the matrix takes: one CTA per SM
    return narrow ? cluster_launch<true>(st, s, a) : cluster_launch<false>(st, s, a);
}

namespace {
// Stored columns of the CTA and of the warp that have most, in both forms, and the
// widest slice.  One thread per CTA and warp of the grid form, then of the cluster.
__global__ void loop_balance_kernel(int nslices, int P, int nw, int clusterSlices, int clusterWarps,
                                    const int* __restrict__ sliceOff, LoopBalance* out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, grid = P * nw;
    const bool cluster = t >= grid;
    int s0, s1, w, W;
    if (!cluster) {
        const int q = t / nw;
        s0 = (int)((int64_t)nslices * q / P), s1 = (int)((int64_t)nslices * (q + 1) / P);
        w = t % nw, W = nw;
    } else {
        const int q = (t - grid) / clusterWarps;
        s0 = min(nslices, q * clusterSlices), s1 = min(nslices, s0 + clusterSlices);
        w = (t - grid) % clusterWarps, W = clusterWarps;
    }
    if (s0 >= s1) return;
    int cols = 0, widest = 0;
    for (int s = s0 + w; s < s1; s += W) {
        const int width = (sliceOff[s + 1] - sliceOff[s]) >> 5;
        cols += width;
        widest = max(widest, width);
    }
    atomicMax(cluster ? &out->clusterWarp : &out->gridWarp, cols);
    if (!cluster) atomicMax(&out->widest, widest);
    if (w == 0) {
        const int all = (sliceOff[s1] - sliceOff[s0]) >> 5;
        atomicMax(cluster ? &out->clusterCols : &out->gridCols, all);
    }
    if (t == 0) out->last = sliceOff[nslices - 1];
}

// Stored entries whose column does not follow that of the lane before: one warp
// per slice.  A row past its last entry counts as on the diagonal.
__global__ void loop_scattered_kernel(int n, int nslices, const int* __restrict__ rowptr, const int* __restrict__ col,
                                      LoopBalance* out) {
    const int lane = threadIdx.x & 31;
    int count = 0;
    for (int s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslices; s += (gridDim.x * blockDim.x) >> 5) {
        const int row = min(32 * s + lane, n - 1);
        const int j0 = rowptr[row], j1 = 32 * s + lane < n ? rowptr[row + 1] : j0;
        const int w = __reduce_max_sync(0xffffffffu, j1 - j0);
        for (int j = 0; j < w; ++j) {
            const int c = j0 + j < j1 ? col[j0 + j] : row;
            const int before = __shfl_up_sync(0xffffffffu, c, 1);
            count += lane > 0 && c != before + 1 ? 1 : 0;
        }
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if (lane == 0 && count > 0) atomicAdd(&out->scattered, count);
}
}  // namespace

cudaError_t cg_loop_balance(cudaStream_t st, int n, int numSms, int64_t stored, const int* sliceOff, const int* rowptr,
                            const int* col, LoopBalance* out) {
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(LoopBalance), st);
    if (e != cudaSuccess) return e;
    const LoopShape g = loop_shape(n, numSms), c = cluster_shape(n);
    const int nslices = (n + 31) / 32, threads = g.P * (g.threads / 32) + c.P * (c.threads / 32);
    loop_balance_kernel<<<(threads + 127) / 128, 128, 0, st>>>(nslices, g.P, g.threads / 32, c.rows / 32, c.threads / 32,
                                                              sliceOff, out);
    if (stored + 7 * (int64_t)n <= kClusterWork)
        loop_scattered_kernel<<<std::max(1, std::min(numSms * 4, (nslices + 3) / 4)), 128, 0, st>>>(n, nslices, rowptr,
                                                                                                  col, out);
    return cudaGetLastError();
}

// A lane owns a row, a CTA an equal number of slices: uneven rows make an
// iteration as long as its longest warp (64 cycles for each column, an FMA of its
// rows' chains) or its fullest CTA (16 cycles, the FP64 pipe).  The graph loop's
// SpMV strides the slices over all SMs, or where the rows are uneven enough for
// every layout to be timed (a padded copy above 1.1 of the entries) gives long rows
// a warp or more.  The one kernel gains 5 - 10 us per iteration elsewhere, so it is
// kept where the surplus is below that.  us per iteration, one kernel / graph, and the
// surplus in 1,000 cycles:
//   all layouts   20,000 rows of 129 at most 19.7 / 31.9 (2), 16^3 with a row of 120
//                 11.6 / 17.8 (7), 2,000 of 100 - 160 19.3 / 19.5 (9), 100,000 of 4 -
//                 60, ascending, 30.6 / 30.5 (5), 20,000 7-point with a row of 300 30.0
//                 / 27.4 (19), 97,000 with 16 of them 33.9 / 19.0 (17), 50,000 with one of
//                 600 50.5 / 28.5 (38), 2,000 rows of 400 - 676 51.9 / 21.3 (39)
//   sliced only   400,000 7-point with a row of 3,000 216 / 627 (0: the graph's kernels
//                 wait for that row too), 7-point and 27-point halves of 48^3 23.1 /
//                 30.8 (8), 60^3 36.1 / 38.3 (15), 76^3 60.3 / 58.7 (29), 648,000
//                 7-point and 64,000 27-point rows 51.9 / 41.4 (42)
// The cluster or the grid: a scattered entry costs the cluster 4.5 cycles of its
// CTA, a column of the longest warp the grid about 130; and the cluster's fullest CTA
// must not lag behind the grid's by more than the 2 us that it gains.  Cluster / grid,
// random rows: 500 of 100 (47,000 scattered) 12.3 / 18.2, 1,000 of 32 (34,000) 9.6 /
// 11.5, of 64 (65,000) 14.8 / 14.0, 2,000 of 16 (36,000) 9.6 / 10.0, of 32 (68,000)
// 14.8 / 11.4, 4,000 of 32 (135,000) 27.5 / 12.0 (graph 17.5); 27-point 16^3 in
// random order (102,000) 21.4 / 10.7, in grid order (15,000) 7.6 / 10.6.
int cg_loop_form(int n, int numSms, int64_t stored, bool allLayouts, const LoopBalance& b) {
    if (!cg_loop_fits(n, numSms)) return 0;
    const int64_t cols = stored / 32, even = 16 * cols / numSms;
    const int64_t grid = std::max<int64_t>(16ll * b.gridCols, 64ll * b.gridWarp);
    const int64_t cluster = std::max<int64_t>(16ll * b.clusterCols, 64ll * b.clusterWarp);
    const int64_t graph = allLayouts ? even : std::max<int64_t>(even, 64ll * b.widest);
    if (grid > graph + (allLayouts ? 8000 : 20000)) return 0;
    if (b.scattered > 27000 + 460 * b.gridWarp || cluster > grid + 16 * cols / kClusterMax + 4000) return 1;
    return cg_cluster_fits(n, stored, b) ? 2 : 1;
}

// The vectors have to fit in shared memory, all but J (1,065,216 rows on 152 SMs; J too up to 856,064).
bool cg_loop_fits(int n, int numSms) { return n > 0 && loop_shape(n, numSms).fixed <= kLoopSmem; }

size_t cg_loop_sync_bytes(int numSms) { return 128 * sizeof(uint32_t) + 3 * sizeof(ulonglong2) * 2 * (size_t)numSms; }

// Steps of 9 where rows of the mean length take fewer of them than of 7: a step
// costs its instructions besides the products, and one with columns to spare
// more (27-point 96^3: 63.4 us per iteration with 9 = 3 steps, 69.1 with 7; 7-point
// 96^3: 40.2 with 9, 33.6 with 7).  Not where a warp has one slice at most, and
// the wait for a step's own loads counts (27-point 32^3: 12.0 with 9, 11.5 with 7).
static int loop_step(int n, int64_t stored, const LoopShape& s) {
    const int64_t rows = ((int64_t)n + 31) / 32 * 32, mean = (stored + rows - 1) / rows;
    const bool fewer = (mean + kStep[1] - 1) / kStep[1] < (mean + kStep[0] - 1) / kStep[0];
    return fewer && s.rows > s.threads ? kStep[1] : kStep[0];
}

cudaError_t cg_loop_launch(cudaStream_t st, int layout, int numSms, int64_t stored, void* sync, LoopArgs a) {
    const LoopShape s = loop_shape(a.n, numSms);
    const int step = loop_step(a.n, stored, s);
    a.nslices = (a.n + 31) / 32;
    a.rows = s.rows;
    a.jOnChip = s.jOnChip ? 1 : 0;
    a.counters = static_cast<uint32_t*>(sync);
    a.posts = reinterpret_cast<ulonglong2*>(a.counters + 128);
    if (layout == 0) return loop_launch_steps<0>(step, st, s, a);
    if (layout == 1) return loop_launch_steps<1>(step, st, s, a);
    return loop_launch_steps<2>(step, st, s, a);
}

}  // namespace xjpcg
