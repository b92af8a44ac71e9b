// The grouped DPD contraction kernel (sm_100a, FP64).
//
// One launch executes every irrep block of a contraction: each CTA owns a
// BM x BN tile of one output block (task) and walks the K segments of that
// task (the irrep assignments of the contracted indices), gathering A / B
// tiles through the planner's stride tables (packed pairs are composite
// indices) into padded shared memory and multiplying them on the FP64
// tensor pipe with mma.sync.m8n8k4.f64 (tcgen05 has no FP64 kind).  K stages
// of 16 are copied with cp.async into a ring, two or three stages ahead of
// the one that is multiplied, one barrier a stage; staging them in registers
// one stage ahead was slower in every shape (twice the time with 128x32 on the
// C1 nmo-71 ladder).  Split-K tiles write
// partial sums that k_splitk_reduce adds in a fixed order, so results are
// deterministic.
#include <atomic>
#include <array>
#include <vector>

#include <map>
#include <memory>
#include <mutex>
#include "runtime.hpp"

namespace cpsd {

namespace {
constexpr int NT = 256, BK = 16, PAD = 4;
// K stages in the ring: four, or three where that lets a third CTA onto the SM
// (four warps with 32 x 32 of the tile each).  The 128x16 tile streams its
// first operand and is better off with the deeper ring (19 columns in 8 irreps
// of 9100 pairs: 1.33 ms with four stages, 1.63 with three).
constexpr int ring(int warps, int bn) { return warps == 4 && bn > 16 ? 3 : 4; }

__device__ __forceinline__ i64 decode1(i64 x, int n, const i64 *ext, const i64 *st) {
    // the last unit takes the remaining quotient whole (x < its extent), so
    // it needs no division; the others divide in 32 bits when both fit
    i64 off = 0;
    for (int u = 0; u < n - 1; u++) {
        const i64 e = ext[u];
        const i64 q = (x <= 0x7fffffffLL && e <= 0x7fffffffLL) ? (i64)((unsigned)x / (unsigned)e) : x / e;
        off += (x - q * e) * st[u];
        x = q;
    }
    return n > 0 ? off + x * st[n - 1] : off;
}

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

template <int BM, int BN, int WARPS>
constexpr int smem_bytes() {
    return (int)sizeof(double) * ring(WARPS, BN) * BK * ((BM + PAD) + (BN + PAD));
}

// 8-byte asynchronous copy, or zero fill without reading the source
__device__ __forceinline__ void stage_cp(double *dst, const double *src, bool read) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(read ? 8 : 0)
                 : "memory");
}
// a table entry by the threads of a CTA, one word each
template <class T>
__device__ __forceinline__ void copy_entry(T *dst, const T *src) {
    static_assert(sizeof(T) % 8 == 0 && sizeof(T) / 8 <= 128, "words of a table entry");
    if (threadIdx.x < sizeof(T) / 8)
        reinterpret_cast<long long *>(dst)[threadIdx.x] = reinterpret_cast<const long long *>(src)[threadIdx.x];
}

template <int BM, int BN, int WM, int WN>
__global__ void __launch_bounds__(32 * WM * WN, WM * WN == 4 ? 3 : 2) k_contract(const double *__restrict__ A, const double *__restrict__ B,
                                                    double *__restrict__ C, const TaskDev *__restrict__ tasks,
                                                    const SegDev *__restrict__ segs, const TileDev *__restrict__ tiles,
                                                    double alpha, double *__restrict__ partial) {
    constexpr int NT = 32 * WM * WN, NST = ring(WM * WN, BN);
    constexpr int WTM = BM / WM, WTN = BN / WN, MI = WTM / 8, NI = WTN / 8;
    constexpr int LA = BM * BK / NT, LB = BN * BK / NT;
    static_assert(LA >= 1 && LB >= 1 && NT % BM == 0 && NT % BK == 0, "tile shape");
    extern __shared__ double dsm[];
    double(*As)[BK][BM + PAD] = reinterpret_cast<double(*)[BK][BM + PAD]>(dsm);
    double(*Bs)[BK][BN + PAD] = reinterpret_cast<double(*)[BK][BN + PAD]>(dsm + NST * BK * (BM + PAD));
    __shared__ i64 offM[BM], offN[BN], offKA[NST][BK], offKB[NST][BK];
    __shared__ TaskDev tk;
    __shared__ SegDev sgs[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp % WM, wn = warp / WM;
    const TileDev tl = tiles[blockIdx.x];
    copy_entry(&tk, tasks + tl.task);
    __syncthreads();
    copy_entry(&sgs[0], segs + tk.seg0);
    const i64 m0 = (i64)tl.mt * BM, n0 = (i64)tl.nt * BN;
    double acc[MI][NI][2];
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NI; j++) acc[i][j][0] = acc[i][j][1] = 0.0;

    for (int si = 0; si < tk.nseg; si++) {
        __syncthreads();
        const SegDev &sg = sgs[si & 1];
        // the next segment's entry travels with this one's first stage
        if (si + 1 < tk.nseg && tid < (int)sizeof(SegDev) / 8)
            stage_cp(reinterpret_cast<double *>(&sgs[(si + 1) & 1]) + tid,
                     reinterpret_cast<const double *>(segs + tk.seg0 + si + 1) + tid, true);
        i64 kb = tl.k_lo - sg.kstart, ke = tl.k_hi - sg.kstart;
        if (kb < 0) kb = 0;
        if (ke > sg.K) ke = sg.K;
        if (kb >= ke) {
            asm volatile("cp.async.wait_all;" ::: "memory");
            continue;
        }
        for (int j = tid; j < BM + BN; j += NT) {
            if (j < BM) {
                const i64 m = m0 + j;
                offM[j] = (m < tk.M) ? sg.baseA + decode1(m, tk.nm, tk.mExt, sg.mSA) : -1;
            } else {
                const i64 n = n0 + j - BM;
                offN[j - BM] = (n < tk.N) ? sg.baseB + decode1(n, tk.nn, tk.nExt, sg.nSB) : -1;
            }
        }
        const int nst = (int)((ke - kb + BK - 1) / BK);
        // operand offsets of index j of K stage s, into ring slot s % NST
        auto decodeK = [&](int s, int j) {
            const i64 k = kb + (i64)s * BK + j;
            i64 a = -1, b = -1;
            if (k < ke) {
                a = b = 0;
                i64 x = k;
                for (int u = 0; u < sg.nk - 1; u++) {
                    const i64 e = sg.kExt[u];
                    const i64 q = (x <= 0x7fffffffLL && e <= 0x7fffffffLL) ? (i64)((unsigned)x / (unsigned)e) : x / e;
                    const i64 r = x - q * e;
                    a += r * sg.kSA[u];
                    b += r * sg.kSB[u];
                    x = q;
                }
                if (sg.nk > 0) {  // the last unit takes the remaining quotient
                    a += x * sg.kSA[sg.nk - 1];
                    b += x * sg.kSB[sg.nk - 1];
                }
            }
            offKA[s % NST][j] = a;
            offKB[s % NST][j] = b;
        };
        // one contracted unit: offsets in a constant step, no table
        const bool afast = sg.aMfast, bfast = sg.bKfast, lin = sg.nk == 1;
        const i64 ksa = sg.kSA[0], ksb = sg.kSB[0];
        // in 32 bits (finish_plan keeps parts below 2^30): bounds and offsets of
        // a stage formed in 64 bits cost the 28 columns of the C1 nmo-71 ladder
        // (128x32) 261 us instead of 231, and a 128x64 ladder 568 instead of 553.
        // The bound as what is left of the range suits the 64-row tiles (C2 nmo-74
        // ladder 352 us, 369 as k0 + k < kend), not the 128-row ones (261, 558)
        const int kend = (int)(ke - kb);
        auto put_a = [&](int buf, int k, int m, i64 om, bool in, i64 ok) {
            stage_cp(&As[buf][k][m], in ? A + om + ok : A, in);
        };
        auto put_b = [&](int buf, int k, int n, i64 on, bool in, i64 ok) {
            stage_cp(&Bs[buf][k][n], in ? B + on + ok : B, in);
        };
        auto issue = [&](int s) {
            if (s < nst) {
                const int buf = s % NST, k0 = s * BK;
                const int at = BM == 64 ? 0 : k0, end = BM == 64 ? kend - k0 : kend;
                if (afast) {  // a thread keeps its row (BM divides NT)
                    const int m = tid % BM;
                    const i64 om = offM[m];
#pragma unroll
                    for (int i = 0; i < LA; i++) {
                        const int k = tid / BM + i * (NT / BM);
                        put_a(buf, k, m, om, om >= 0 && at + k < end, lin ? (kb + k0 + k) * ksa : offKA[buf][k]);
                    }
                } else {  // a thread keeps its contracted index
                    const int k = tid % BK;
                    const i64 ok = lin ? (kb + k0 + k) * ksa : offKA[buf][k];
#pragma unroll
                    for (int i = 0; i < LA; i++) {
                        const int m = tid / BK + i * (NT / BK);
                        const i64 om = offM[m];
                        put_a(buf, k, m, om, om >= 0 && at + k < end, ok);
                    }
                }
                if (bfast) {
                    const int k = tid % BK;
                    const i64 ok = lin ? (kb + k0 + k) * ksb : offKB[buf][k];
#pragma unroll
                    for (int i = 0; i < LB; i++) {
                        const int n = tid / BK + i * (NT / BK);
                        const i64 on = offN[n];
                        put_b(buf, k, n, on, on >= 0 && at + k < end, ok);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < LB; i++) {
                        const int e = tid + i * NT, n = e % BN, k = e / BN;
                        const i64 on = offN[n];
                        put_b(buf, k, n, on, on >= 0 && at + k < end, lin ? (kb + k0 + k) * ksb : offKB[buf][k]);
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");  // an empty group past the end keeps the count
        };
        if (!lin && tid < BK * NST) decodeK(tid / BK, tid % BK);
        __syncthreads();
#pragma unroll
        for (int s = 0; s < NST - 1; s++) issue(s);
        for (int s = 0; s < nst; s++) {
            asm volatile("cp.async.wait_group %0;" ::"n"(NST - 2) : "memory");
            __syncthreads();  // stage s is complete; slot s - 1 and its offsets are free
            issue(s + NST - 1);
            if (!lin && tid < BK && s + NST < nst) decodeK(s + NST, tid);
            const int buf = s % NST;
#pragma unroll
            for (int kk = 0; kk < BK / 4; kk++) {
                const int kr = kk * 4 + (lane & 3);
                double a[MI], b[NI];
#pragma unroll
                for (int i = 0; i < MI; i++) a[i] = As[buf][kr][wm * WTM + i * 8 + (lane >> 2)];
#pragma unroll
                for (int j = 0; j < NI; j++) b[j] = Bs[buf][kr][wn * WTN + j * 8 + (lane >> 2)];
#pragma unroll
                for (int i = 0; i < MI; i++)
#pragma unroll
                    for (int j = 0; j < NI; j++) dmma(acc[i][j], a[i], b[j]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int rl = lane >> 2, cl = 2 * (lane & 3);
    if (tl.part >= 0) {
        double *P = partial + (size_t)tl.part * (BM * BN);
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NI; j++) {
                int r = wm * WTM + i * 8 + rl, c = wn * WTN + j * 8 + cl;
                P[r * BN + c] = acc[i][j][0];
                P[r * BN + c + 1] = acc[i][j][1];
            }
        return;
    }
    for (int j = tid; j < BM + BN; j += NT) {
        if (j < BM) {
            const i64 m = m0 + j;
            offM[j] = (m < tk.M) ? tk.baseC + decode1(m, tk.nm, tk.mExt, tk.mSC) : -1;
        } else {
            const i64 n = n0 + j - BM;
            offN[j - BM] = (n < tk.N) ? decode1(n, tk.nn, tk.nExt, tk.nSC) : -1;
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < MI; i++) {
        i64 om = offM[wm * WTM + i * 8 + rl];
        if (om < 0) continue;
#pragma unroll
        for (int j = 0; j < NI; j++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                i64 on = offN[wn * WTN + j * 8 + cl + h];
                if (on < 0) continue;
                C[om + on] += alpha * acc[i][j][h];
            }
    }
}

// Sum the split-K partial tiles of the output tiles in a fixed order.  One
// thread per tile element: block b covers elements [NT*(b % chunks), +NT)
// of reduce group b / chunks (chunks = bm*bn / NT), with four independent
// partial sums so that the loads of several partial tiles are in flight.
__global__ void __launch_bounds__(NT) k_splitk_reduce(const int *__restrict__ red, const TaskDev *__restrict__ tasks,
                                                      const double *__restrict__ partial, double *__restrict__ C,
                                                      double alpha, int bm, int bn) {
    const int chunks = bm * bn / NT;
    const int *r = red + 5 * (blockIdx.x / chunks);
    const int e = (blockIdx.x % chunks) * NT + threadIdx.x;
    const TaskDev &tk = tasks[r[0]];
    const i64 m = (i64)r[1] * bm + e / bn, n = (i64)r[2] * bn + e % bn;
    if (m >= tk.M || n >= tk.N) return;
    const i64 p0 = r[3];
    const int ns = r[4];
    const size_t ts = (size_t)bm * bn;
    const double *P = partial + (size_t)p0 * ts + e;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int q = 0;
    for (; q + 4 <= ns; q += 4) {
        s0 += P[(size_t)q * ts];
        s1 += P[(size_t)(q + 1) * ts];
        s2 += P[(size_t)(q + 2) * ts];
        s3 += P[(size_t)(q + 3) * ts];
    }
    for (; q < ns; q++) s0 += P[(size_t)q * ts];
    const double s = (s0 + s1) + (s2 + s3);
    C[tk.baseC + decode1(m, tk.nm, tk.mExt, tk.mSC) + decode1(n, tk.nn, tk.nExt, tk.nSC)] += alpha * s;
}

// optional CUDA-event timing of every contraction launch (on its stream)
struct Timing {
    bool on = false;
    std::vector<cudaEvent_t> pool;
    size_t used = 0;
    std::vector<double> flops;
    std::vector<std::array<int64_t, 4>> shape;  // tasks, segments, tiles, tile config
};
Timing &timing() {
    thread_local Timing t;
    return t;
}
int timing_event(cudaEvent_t *e) {
    Timing &t = timing();
    if (t.used == t.pool.size()) {
        cudaEvent_t ev;
        CPSD_TRY(cuda_check(cudaEventCreate(&ev), "event create"));
        t.pool.push_back(ev);
    }
    *e = t.pool[t.used++];
    return CPSD_OK;
}
}  // namespace

const int TILE_BM[NTILE] = {128, 128, 64, 64, 128};
const int TILE_BN[NTILE] = {64, 32, 128, 64, 16};

int contract_timing(int enable) {
    timing().on = enable != 0;
    return CPSD_OK;
}
bool contract_timing_on() { return timing().on; }

int timing_begin(double flops, int64_t a, int64_t b, int64_t c, int64_t kind, cudaEvent_t *end) {
    *end = nullptr;
    if (!timing().on) return CPSD_OK;
    cudaEvent_t e0;
    CPSD_TRY(timing_event(&e0));
    CPSD_TRY(timing_event(end));
    timing().flops.push_back(flops);
    timing().shape.push_back({a, b, c, kind});
    return cuda_check(cudaEventRecord(e0, stream()), "event record");
}

int timing_end(cudaEvent_t end) {
    if (!end) return CPSD_OK;
    return cuda_check(cudaEventRecord(end, stream()), "event record");
}

int contract_records(double *ms, double *flops, int64_t *shape, int64_t maxrec, int64_t *nrec) {
    Timing &t = timing();
    int64_t n = 0;
    for (size_t i = 0; i + 1 < t.used && n < maxrec; i += 2, n++) {
        CPSD_TRY(cuda_check(cudaEventSynchronize(t.pool[i + 1]), "event sync"));
        float x = 0.f;
        CPSD_TRY(cuda_check(cudaEventElapsedTime(&x, t.pool[i], t.pool[i + 1]), "event time"));
        ms[n] = x;
        flops[n] = t.flops[i / 2];
        for (int k = 0; k < 4; k++) shape[4 * n + k] = t.shape[i / 2][k];
    }
    *nrec = n;
    return CPSD_OK;
}

int contract_time(double *ms, int64_t *launches, double *flops, int reset) {
    Timing &t = timing();
    double tot = 0.0, fl = 0.0;
    for (size_t i = 0; i + 1 < t.used; i += 2) {
        if (t.shape[i / 2][3] >= 30) continue;  // solver / layout records are not contraction work
        CPSD_TRY(cuda_check(cudaEventSynchronize(t.pool[i + 1]), "event sync"));
        float x = 0.f;
        CPSD_TRY(cuda_check(cudaEventElapsedTime(&x, t.pool[i], t.pool[i + 1]), "event time"));
        tot += x;
        fl += t.flops[i / 2];
    }
    if (ms) *ms = tot;
    if (launches) *launches = (int64_t)(t.used / 2);
    if (flops) *flops = fl;
    if (reset) {
        t.used = 0;
        t.flops.clear();
        t.shape.clear();
    }
    return CPSD_OK;
}

namespace {
// the empirical tile-shape choice: per plan, the variant that ran fastest
std::atomic<int> g_autotune{0};
std::atomic<int64_t> g_tuned{0}, g_changed{0};
std::mutex &tune_mutex() {
    static std::mutex m;
    return m;
}
std::map<const ContractPlan *, const ContractPlan *> &tuned_plans() {
    static std::map<const ContractPlan *, const ContractPlan *> m;
    return m;
}
std::vector<std::unique_ptr<ContractPlan>> &tuned_variants() {
    static std::vector<std::unique_ptr<ContractPlan>> v;
    return v;
}
// one past the largest output offset a plan writes
i64 plan_c_extent(const ContractPlan *p) {
    i64 hi = 0;
    for (const TaskDev &t : p->h_tasks) {
        i64 e = t.baseC;
        for (int u = 0; u < t.nm; u++) e += (t.mExt[u] - 1) * t.mSC[u];
        for (int u = 0; u < t.nn; u++) e += (t.nExt[u] - 1) * t.nSC[u];
        hi = std::max(hi, e + 1);
    }
    return hi;
}
int launch_tiles(const ContractPlan *p, const double *A, const double *B, double *C, double alpha);
// the fastest of the four tile shapes for plan p, timed on a scratch output
int tune_plan(const ContractPlan *p, const double *A, const double *B, const ContractPlan **best) {
    *best = p;
    const i64 n = plan_c_extent(p);
    ScratchScope sc;
    double *Ct;
    CPSD_TRY(scratch(n, &Ct));
    CPSD_TRY(cuda_check(cudaMemsetAsync(Ct, 0, sizeof(double) * (size_t)n, stream()), "tune scratch"));
    cudaEvent_t e0, e1;
    CPSD_TRY(cuda_check(cudaEventCreate(&e0), "event"));
    CPSD_TRY(cuda_check(cudaEventCreate(&e1), "event"));
    float best_ms = 1e30f;
    int rc = CPSD_OK;
    for (int c = 0; c < NTILE - 1 && rc == CPSD_OK; c++) {
        const ContractPlan *q = p;
        if (c != p->cfg) {
            auto v = std::make_unique<ContractPlan>();
            v->flops = p->flops;
            v->task_mkey = p->task_mkey;
            v->task_nkey = p->task_nkey;
            v->seg_kkey = p->seg_kkey;
            finish_plan(v.get(), p->h_tasks, p->h_segs, c);
            q = v.get();
            tuned_variants().push_back(std::move(v));
        }
        float ms = 0.f;
        for (int rep = 0; rep < 2 && rc == CPSD_OK; rep++) {  // the second run is timed
            rc = cuda_check(cudaEventRecord(e0, stream()), "event record");
            if (rc == CPSD_OK) rc = launch_tiles(q, A, B, Ct, 1.0);
            if (rc == CPSD_OK) rc = cuda_check(cudaEventRecord(e1, stream()), "event record");
            if (rc == CPSD_OK) rc = cuda_check(cudaEventSynchronize(e1), "event sync");
            if (rc == CPSD_OK) rc = cuda_check(cudaEventElapsedTime(&ms, e0, e1), "event time");
        }
        if (rc == CPSD_OK && ms < best_ms * 0.97f) {  // the cost model's shape unless 3 % faster
            best_ms = ms;
            *best = q;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return rc;
}
}  // namespace

int set_tile_autotune(int on) {
    g_autotune.store(on ? 1 : 0);
    return CPSD_OK;
}
int tile_autotune_stats(int64_t *tuned, int64_t *changed) {
    if (tuned) *tuned = g_tuned.load();
    if (changed) *changed = g_changed.load();
    return CPSD_OK;
}

int launch_contract(const ContractPlan *p, const double *A, const double *B, double *C, double alpha) {
    if (p->empty) return CPSD_OK;
    if (g_autotune.load()) {
        const ContractPlan *q = nullptr;
        {
            std::lock_guard<std::mutex> lock(tune_mutex());
            auto it = tuned_plans().find(p);
            if (it != tuned_plans().end()) q = it->second;
        }
        if (!q) {
            std::lock_guard<std::mutex> lock(tune_mutex());
            CPSD_TRY(tune_plan(p, A, B, &q));
            tuned_plans()[p] = q;
            g_tuned++;
            if (q != p) g_changed++;
        }
        p = q;
    }
    return launch_tiles(p, A, B, C, alpha);
}

namespace {
// kernel attributes of the tile shapes (of the current device when `again`)
int tile_attrs(bool again = false) {
    static std::atomic<bool> done{false};
    if (done.load(std::memory_order_acquire) && !again) return CPSD_OK;
    auto one = [](const void *k, int bytes) {
        return cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), "smem attr");
    };
    CPSD_TRY(one((const void *)k_contract<128, 64, 4, 2>, smem_bytes<128, 64, 8>()));
    CPSD_TRY(one((const void *)k_contract<128, 32, 4, 1>, smem_bytes<128, 32, 4>()));
    CPSD_TRY(one((const void *)k_contract<64, 128, 2, 4>, smem_bytes<64, 128, 8>()));
    CPSD_TRY(one((const void *)k_contract<64, 64, 2, 2>, smem_bytes<64, 64, 4>()));
    CPSD_TRY(one((const void *)k_contract<128, 16, 4, 1>, smem_bytes<128, 16, 4>()));
    done.store(true, std::memory_order_release);
    return CPSD_OK;
}
void run_tiles(int cfg, int ntiles, const double *A, const double *B, double *C, const TaskDev *tk, const SegDev *sg,
               const TileDev *tl, double alpha, double *part) {
#define CPSD_TILE(BM, BN, WM, WN)                                                                                \
    k_contract<BM, BN, WM, WN><<<ntiles, 32 * WM * WN, smem_bytes<BM, BN, WM * WN>(), stream()>>>(A, B, C, tk, sg, tl, alpha, part)
    switch (cfg) {
    case 0: CPSD_TILE(128, 64, 4, 2); break;
    case 1: CPSD_TILE(128, 32, 4, 1); break;
    case 2: CPSD_TILE(64, 128, 2, 4); break;
    case 3: CPSD_TILE(64, 64, 2, 2); break;
    default: CPSD_TILE(128, 16, 4, 1); break;
    }
#undef CPSD_TILE
}

int launch_tiles(const ContractPlan *p, const double *A, const double *B, double *C, double alpha) {
    CPSD_TRY(const_cast<ContractPlan *>(p)->upload());
    const int bm = TILE_BM[p->shape()], bn = TILE_BN[p->shape()];
    double *part = nullptr;
    ScratchScope scope;
    if (p->nparts > 0) {
        const int rc = scratch(p->nparts * bm * bn, &part);
        // a caller's workspace may hold no more than the fixed rule asks for
        // (K parts of 256 and more): the same contraction with those tiles
        const ContractPlan *q = nullptr;
        if (rc != CPSD_OK && arena().external && plan_fixed(p, &q) == CPSD_OK &&
            q->nparts * TILE_BM[q->shape()] * TILE_BN[q->shape()] < p->nparts * bm * bn)
            return launch_tiles(q, A, B, C, alpha);
        CPSD_TRY(rc);
    }
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (timing().on) {
        CPSD_TRY(timing_event(&e0));
        CPSD_TRY(timing_event(&e1));
        timing().flops.push_back(p->flops);
        timing().shape.push_back({p->ntasks, p->nsegs, p->ntiles, p->cfg});
        CPSD_TRY(cuda_check(cudaEventRecord(e0, stream()), "event record"));
    }
    CPSD_TRY(tile_attrs());
    run_tiles(p->shape(), p->ntiles, A, B, C, p->d_tasks, p->d_segs, p->d_tiles, alpha, part);
    count_launch();
    ctx().flops += p->flops;
    if (e1) CPSD_TRY(cuda_check(cudaEventRecord(e1, stream()), "event record"));
    if (p->nreduce > 0) {
        k_splitk_reduce<<<p->nreduce * (bm * bn / NT), NT, 0, stream()>>>(p->d_reduce, p->d_tasks, part, C, alpha,
                                                                          bm, bn);
        count_launch();
    }
    return cuda_check(cudaGetLastError(), "k_contract");
}
}  // namespace

// ------------------------------------------- contraction without allocation
// Some callers may not allocate device memory while they run a contraction:
// a host program that hands (nearly) all of HBM to its own pool at start-up
// sees cudaMalloc fail, and cudaMalloc / cudaFree can stall the device in
// the middle of a time-critical loop.  For them, launch_contract_noalloc
// keeps the plan tables and the split-K partial tiles in one fixed region
// compiled into this library instead of the cudaMalloc'ed plan copies and
// the scratch arena launch_contract uses.  Limits and rules:
//  - the region holds CPSD_NOALLOC_SCRATCH_BYTES; a contraction whose
//    tables plus partial tiles need more is rejected (CPSD_EARG) before any
//    work is queued;
//  - nothing in the region has to start at zero: every word a call reads
//    was written earlier in the same call (tables copied in, partial tiles
//    stored in full before the reduce reads them);
//  - there is one region per device, so two calls whose work overlaps in
//    time (different streams, or host threads) race on it; calls queued on
//    one stream are ordered and safe;
//  - the first call on each device does the set-up (symbol address of the
//    region, kernel attributes); make that first call before any stream
//    capture begins;
//  - the plan tables are copied from the plan's pageable host vectors
//    (pinned staging would itself be an allocation); CUDA lets such a copy
//    start only after the work queued earlier on the stream, so a call can
//    block the host until then.
namespace {
__device__ __align__(256) unsigned char g_noalloc_scratch[CPSD_NOALLOC_SCRATCH_BYTES];

constexpr int NOALLOC_MAXDEV = 64;
// region address per device ordinal (null until set up); the set-up runs
// under a lock so that two host threads' first calls do not race on it
std::atomic<unsigned char *> g_noalloc_base[NOALLOC_MAXDEV];
std::mutex g_noalloc_setup_mutex;

int noalloc_setup(unsigned char **base) {
    int dev = 0;
    CPSD_TRY(cuda_check(cudaGetDevice(&dev), "cudaGetDevice"));
    if (dev < 0 || dev >= NOALLOC_MAXDEV) return set_error(CPSD_EARG, "device ordinal beyond 63");
    if (!g_noalloc_base[dev].load()) {
        std::lock_guard<std::mutex> lock(g_noalloc_setup_mutex);
        if (g_noalloc_base[dev].load()) {
            *base = g_noalloc_base[dev].load();
            return CPSD_OK;
        }
        void *p = nullptr;
        CPSD_TRY(cuda_check(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress(noalloc scratch)"));
        CPSD_TRY(tile_attrs(true));
        g_noalloc_base[dev].store((unsigned char *)p);
    }
    *base = g_noalloc_base[dev].load();
    return CPSD_OK;
}

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
}  // namespace

size_t contract_noalloc_bytes(const ContractPlan *plan) {
    if (plan->empty) return 0;
    const ContractPlan *p;
    if (plan_fixed(plan, &p) != CPSD_OK) return 0;
    const size_t tile = (size_t)TILE_BM[p->cfg] * TILE_BN[p->cfg] * sizeof(double);
    return align256(p->h_tasks.size() * sizeof(TaskDev)) + align256(p->h_segs.size() * sizeof(SegDev)) +
           align256(p->h_tiles.size() * sizeof(TileDev)) + align256(p->h_reduce.size() * sizeof(int)) +
           align256((size_t)p->nparts * tile);
}

int launch_contract_noalloc(const ContractPlan *plan, const double *A, const double *B, double *C, double alpha) {
    if (plan->empty) return CPSD_OK;
    const size_t need = contract_noalloc_bytes(plan);
    const ContractPlan *p;
    CPSD_TRY(plan_fixed(plan, &p));
    if (need > (size_t)CPSD_NOALLOC_SCRATCH_BYTES)
        return set_error(CPSD_EARG, "contraction needs " + std::to_string(need) +
                                        " bytes of scratch; the no-allocation entry point holds at most " +
                                        std::to_string((size_t)CPSD_NOALLOC_SCRATCH_BYTES));
    unsigned char *base = nullptr;
    CPSD_TRY(noalloc_setup(&base));
    size_t off = 0;
    auto place = [&](const void *src, size_t bytes, void **dst) -> int {
        *dst = base + off;
        off += align256(bytes);
        if (bytes == 0) return CPSD_OK;
        return cuda_check(cudaMemcpyAsync(*dst, src, bytes, cudaMemcpyHostToDevice, stream()), "copy plan tables");
    };
    void *d_tasks, *d_segs, *d_tiles, *d_reduce;
    CPSD_TRY(place(p->h_tasks.data(), p->h_tasks.size() * sizeof(TaskDev), &d_tasks));
    CPSD_TRY(place(p->h_segs.data(), p->h_segs.size() * sizeof(SegDev), &d_segs));
    CPSD_TRY(place(p->h_tiles.data(), p->h_tiles.size() * sizeof(TileDev), &d_tiles));
    CPSD_TRY(place(p->h_reduce.data(), p->h_reduce.size() * sizeof(int), &d_reduce));
    double *part = p->nparts > 0 ? (double *)(base + off) : nullptr;
    const TaskDev *tk = (const TaskDev *)d_tasks;
    const SegDev *sg = (const SegDev *)d_segs;
    const TileDev *tl = (const TileDev *)d_tiles;
    const int bm = TILE_BM[p->cfg], bn = TILE_BN[p->cfg];
    cudaEvent_t e0 = nullptr, e1 = nullptr;  // timing records, as launch_contract keeps them
    if (timing().on) {
        CPSD_TRY(timing_event(&e0));
        CPSD_TRY(timing_event(&e1));
        timing().flops.push_back(p->flops);
        timing().shape.push_back({p->ntasks, p->nsegs, p->ntiles, p->cfg});
        CPSD_TRY(cuda_check(cudaEventRecord(e0, stream()), "event record"));
    }
    run_tiles(p->cfg, p->ntiles, A, B, C, tk, sg, tl, alpha, part);
    count_launch();
    ctx().flops += p->flops;
    if (e1) CPSD_TRY(cuda_check(cudaEventRecord(e1, stream()), "event record"));
    if (p->nreduce > 0) {
        k_splitk_reduce<<<p->nreduce * (bm * bn / NT), NT, 0, stream()>>>((const int *)d_reduce, tk, part, C, alpha,
                                                                          bm, bn);
        count_launch();
    }
    return cuda_check(cudaGetLastError(), "k_contract (no allocation)");
}

}  // namespace cpsd
