// Packed pairs times singles vectors (see pairblk.cuh).
//
// The list is read once and bounds the work: 8 bytes for 4 nj flops.  A warp
// takes one irrep block of one column, a strip of 8 second indices q at a
// time: the strip's contiguous runs of p go to shared memory with 8-byte
// cp.async, a strip ahead, zero-filled where the packed triangle or the block
// ends.  Both products of a stored element come from that one copy, as FP64
// tensor instructions with the roots' columns j as their N = 8: the sums over
// q stay in registers for the whole block, those over p are finished within
// the strip.  Strips have a leading dimension of 4 mod 16 doubles, so that
// both fragment shapes (8 p x 4 q and 8 q x 4 p) fall on different banks.
// A warp only reads what it copied itself.  C2v nmo 151 (373 MB of list): 151 us a
// call; 210 us with the copies' addresses formed anew for every element (64
// instructions per 32 elements, issue-bound) and the strip's other loads not
// ahead; expansion and row-dot contraction took 813 us.
#include <algorithm>
#include <map>
#include <mutex>

#include "pairblk.cuh"

namespace cpsd {

namespace {

constexpr int PW = 4;   // warps per CTA
constexpr int PST = 2;  // strips in flight per warp

__device__ __forceinline__ void pb_dmma(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// 8-byte copy, or zero fill without reading the source
__device__ __forceinline__ void pb_cp(uint32_t dst, const double *src, bool read) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(read ? 8 : 0) : "memory");
}

template <int FT>
constexpr int pb_ld() {
    return FT * 8 + 4;  // FT a multiple of 4: 4 mod 16
}
template <int FT>
constexpr int pb_strip() {
    return 8 * pb_ld<FT>();
}

// this lane's columns of one group of eight: column = j + nj root
struct PbCols {
    i64 rq, rp;        // r of column c0 + (lane >> 2): -1 when there is none
    i64 op[2], oq[2];  // out of columns c0 + 2 (lane & 3) + {0, 1}
};
__device__ __forceinline__ i64 pb_col(int c, int nj, int nb, i64 sj, i64 sb) {
    if (c >= nj * nb) return -1;
    const int root = c / nj, j = c - root * nj;
    return j * sj + root * sb;
}

// one block of one column: V its first element, r and out the operands with
// this column's offsets added (rq, rp, op, oq of cl are column offsets)
template <int FT>
__device__ void pb_block(const PairGroup &g, const double *__restrict__ V, const double *__restrict__ rq,
                         const double *__restrict__ rp, double *op, double *oq, i64 os, const PbCols &cl, double ap,
                         double aq, double *ring) {
    constexpr int LD = pb_ld<FT>();
    const int lane = threadIdx.x & 31, hi = lane >> 2, lo = lane & 3;
    const bool dop = g.ncp > 0, doq = g.ncq > 0;
    const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring + lane);
    for (int p0 = 0; p0 < g.np; p0 += FT * 8) {
        const int np = min(FT * 8, g.np - p0);
        double acc[FT][2], bp[2 * FT];
#pragma unroll
        for (int t = 0; t < FT; t++) acc[t][0] = acc[t][1] = 0.0;
#pragma unroll
        for (int t = 0; t < 2 * FT; t++) {
            const int p = 4 * t + lo;
            bp[t] = doq && cl.rp >= 0 && p < np ? __ldg(rp + cl.rp + p0 + p) : 0.0;
        }
        // the triangle's strips left of p0 hold nothing of this row chunk
        const int s0 = g.tri ? p0 / 8 : 0, s1 = (g.nq + 7) / 8;
        auto rows = [&](int s) {  // rows of strip s, rounded up to 8
            const int lim = g.tri ? min(np, 8 * s + 7 - p0) : np;
            return lim <= 0 ? 0 : (lim + 7) & ~7;
        };
        // whole runs of 32 rows, zero-filled past the strip's last row (a
        // strip is FT * 8 rows wide, a multiple of 32); addresses go on by the
        // length of a run, three or four instructions a copy
        auto issue = [&](int s) {
            if (s < s1) {
                const int pr = rows(s), q0 = 8 * s;
                uint32_t d = ring_at + (uint32_t)((s % PST) * pb_strip<FT>()) * 8;
                const double *src = V + (g.tri ? (i64)q0 * (q0 - 1) / 2 : (i64)q0 * g.np) + p0 + lane;
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int q = q0 + e, lim = (q < g.nq ? (g.tri ? min(np, q - p0) : np) : 0) - lane;
#pragma unroll
                    for (int i = 0; i < FT / 4; i++)
                        if (32 * i < pr) pb_cp(d + 256 * i, 32 * i < lim ? src + 32 * i : V, 32 * i < lim);
                    src += g.tri ? q : g.np;
                    d += LD * 8;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int i = 0; i < PST - 1; i++) issue(s0 + i);
        // r of the strip's rows q and the old outputs of its q product, a strip
        // ahead like the copies
        double bq[2], old[2], bqn[2], oldn[2];
        auto fetch = [&](int s, double (&b)[2], double (&o)[2]) {
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int q = 8 * s + 4 * i + lo;
                b[i] = dop && cl.rq >= 0 && q < g.nq ? __ldg(rq + cl.rq + q) : 0.0;
                o[i] = doq && cl.oq[i] >= 0 && 8 * s + hi < g.nq ? oq[cl.oq[i] + (8 * s + hi) * os] : 0.0;
            }
        };
        fetch(s0, bq, old);
        for (int s = s0; s < s1; s++) {
            issue(s + PST - 1);
            const int q0 = 8 * s, pr = rows(s);
            fetch(s + 1, bqn, oldn);
            asm volatile("cp.async.wait_group %0;" ::"n"(PST - 1) : "memory");
            __syncwarp();
            const double *d = ring + (s % PST) * pb_strip<FT>();
            if (dop) {
#pragma unroll
                for (int t = 0; t < FT; t++)
                    if (8 * t < pr) {
                        pb_dmma(acc[t], d[lo * LD + 8 * t + hi], bq[0]);
                        pb_dmma(acc[t], d[(4 + lo) * LD + 8 * t + hi], bq[1]);
                    }
            }
            if (doq) {
                double c0[2] = {0.0, 0.0}, c1[2] = {0.0, 0.0};
#pragma unroll
                for (int t = 0; t < FT; t++)
                    if (8 * t < pr) {
                        pb_dmma(c0, d[hi * LD + 8 * t + lo], bp[2 * t]);
                        pb_dmma(c1, d[hi * LD + 8 * t + 4 + lo], bp[2 * t + 1]);
                    }
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (cl.oq[i] >= 0 && q0 + hi < g.nq) oq[cl.oq[i] + (q0 + hi) * os] = old[i] + aq * (c0[i] + c1[i]);
            }
#pragma unroll
            for (int i = 0; i < 2; i++) {
                bq[i] = bqn[i];
                old[i] = oldn[i];
            }
            __syncwarp();  // the strip's slot is copied to again
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (dop) {
            double old[FT][2];
#pragma unroll
            for (int t = 0; t < FT; t++)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    old[t][i] = cl.op[i] >= 0 && 8 * t + hi < np ? op[cl.op[i] + (p0 + 8 * t + hi) * os] : 0.0;
#pragma unroll
            for (int t = 0; t < FT; t++)
#pragma unroll
                for (int i = 0; i < 2; i++)
                    if (cl.op[i] >= 0 && 8 * t + hi < np)
                        op[cl.op[i] + (p0 + 8 * t + hi) * os] = old[t][i] + ap * acc[t][i];
        }
    }
}

// W(em,bj): a warp per (block, b, m, column group); the column groups of one
// block are neighbours, so the list is read from memory once
template <int FT>
__global__ void __launch_bounds__(PW * 32, 3) k_pair_wmbej(const PairGroup *__restrict__ groups, int ngroups, i64 items,
                                                        int ncg, const double *__restrict__ V,
                                                        const double *__restrict__ r, double *__restrict__ W, double f,
                                                        int nb, i64 rb, i64 wb) {
    extern __shared__ double pb_ring[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const i64 it = (i64)blockIdx.x * PW + warp;
    if (it >= items * ncg) return;
    const int item = (int)(it / ncg), c0 = (int)(it - (i64)item * ncg) * 8;
    int lo = 0, hi = ngroups - 1;  // last group starting at or before item
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (groups[mid].start <= item) lo = mid;
        else hi = mid - 1;
    }
    const PairGroup g = groups[lo];
    if (c0 >= max(g.ncp, g.ncq) * nb) return;
    const int m = (item - g.start) / g.nx, x = item - g.start - m * g.nx;
    PbCols cl;
    cl.rq = pb_col(c0 + (lane >> 2), g.ncp, nb, g.rqj, rb);
    cl.rp = pb_col(c0 + (lane >> 2), g.ncq, nb, g.rpj, rb);
#pragma unroll
    for (int i = 0; i < 2; i++) {
        cl.op[i] = pb_col(c0 + 2 * (lane & 3) + i, g.ncp, nb, g.opj, wb);
        cl.oq[i] = pb_col(c0 + 2 * (lane & 3) + i, g.ncq, nb, g.oqj, wb);
    }
    pb_block<FT>(g, V + g.v + x * g.vx + m * g.vm, r + g.rq, r + g.rp, W + g.op + x * g.opx + m * g.opm,
                 W + g.oq + x * g.oqx + m * g.oqm, 1, cl, -f, f, pb_ring + warp * PST * pb_strip<FT>());
}

// F(a,e): a CTA per row a, its warps sharing the (m, irrep of m) columns;
// each warp sums its columns in shared memory, then the warps' sums are added
// in order
template <int FT>
__global__ void __launch_bounds__(PW * 32, 3) k_pair_fae(const PairGroup *__restrict__ groups,
                                                      const int *__restrict__ glist, const int *__restrict__ rowirr,
                                                      const double *__restrict__ V, const double *__restrict__ r,
                                                      double *__restrict__ F, double f, int c0, int nb, i64 rb, i64 fb,
                                                      int maxe) {
    extern __shared__ double pb_ring[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ha = rowirr[2 * blockIdx.x], a = rowirr[2 * blockIdx.x + 1];
    const int g0 = glist[ha], g1 = glist[ha + 1];
    if (g0 == g1) return;
    const int nc = min(8, nb - c0);  // roots of this launch
    double *sums = pb_ring + PW * PST * pb_strip<FT>(), *mine = sums + (size_t)warp * maxe * 8;
    for (int e = lane; e < maxe * 8; e += 32) mine[e] = 0.0;
    __syncwarp();
    PbCols cl;
    cl.rq = cl.rp = (lane >> 2) < nc ? (c0 + (lane >> 2)) * rb : -1;
#pragma unroll
    for (int i = 0; i < 2; i++) {
        const int c = 2 * (lane & 3) + i;
        cl.op[i] = cl.oq[i] = c < nc ? c : -1;
    }
    int col = 0, ne = 0;
    i64 out = 0, os = 0;
    for (int k = g0; k < g1; k++) {
        const PairGroup g = groups[k];
        ne = g.ncp > 0 ? g.np : g.nq;
        out = g.op + a * g.opx;
        os = g.opj;  // stride of e in F
        for (int m = 0; m < g.nm; m++, col++) {
            if (col % PW != warp) continue;
            pb_block<FT>(g, V + g.v + a * g.vx + m * g.vm, r + g.rq + m * g.rqm, r + g.rp + m * g.rpm, mine, mine, 8,
                         cl, f, -f, pb_ring + warp * PST * pb_strip<FT>());
            __syncwarp();
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < ne * nc; e += PW * 32) {
        const int c = e / ne, i = e - c * ne;
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < PW; w++) v += sums[((size_t)w * maxe + i) * 8 + c];
        F[out + i * os + (c0 + c) * fb] += v;
    }
}

bool same_pop(const i64 *a, const i64 *b) { return std::equal(a, a + 8, b); }
bool is_zorb8(const i64 *p) { return same_pop(p, ZORB); }

// a packed (p<q | x m) list of irrep 1 and a singles vector (q m' | ..)
bool layouts_ok(const Ten &V, const Ten &r) {
    const Desc &v = V.d, &s = r.d;
    return v.sym == 1 && v.iop[0] == 0 && v.iop[1] == 1 && V.bs == 0 && same_pop(v.pop[0], v.pop[1]) &&
           same_pop(v.pop[0], v.pop[2]) && s.iop[0] == 1 && s.iop[1] == 1 && same_pop(s.pop[0], v.pop[0]) &&
           same_pop(s.pop[1], v.pop[3]) && is_zorb8(s.pop[2]) && is_zorb8(s.pop[3]);
}

// offset of the irrep (hp, hq) block in the packed pair space of its irrep
i64 pair_off(const Desc &v, i64 hq, i64 h) { return isymoffso(hq, h, v.pop[0], v.pop[1], 0) - 1; }
// (row of irrep ha, column j = 0 of irrep hj) of a two-index vector
i64 vec_off(const Desc &s, i64 hj) { return isymoffso(hj, s.sym, s.pop[0], s.pop[1], 1) - 1; }

template <class Build>
int cached(std::map<std::string, std::unique_ptr<PairBlkPlan>> &cache, std::mutex &mx, const std::string &key,
           PairBlkPlan **out, Build build) {
    std::lock_guard<std::mutex> lock(mx);
    auto &p = cache[key];
    if (!p) {
        p = std::make_unique<PairBlkPlan>();
        build(*p);
    }
    *out = p.get();
    return CPSD_OK;
}

template <int FT>
int pb_attr(const void *k, size_t smem, std::atomic<bool> &done) {
    if (done.load(std::memory_order_acquire)) return CPSD_OK;
    CPSD_TRY(cuda_check(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                        "pair kernel smem attr"));
    done.store(true, std::memory_order_release);
    return CPSD_OK;
}
template <int FT>
constexpr size_t pb_smem() {
    return sizeof(double) * PW * PST * pb_strip<FT>();
}

template <int FT>
int wmbej_go(const PairBlkPlan &p, const Ten &V, const Ten &r, Ten &W, double f, i64 nb, i64 wb) {
    static std::atomic<bool> attr{false};
    CPSD_TRY(pb_attr<FT>((const void *)k_pair_wmbej<FT>, pb_smem<FT>(), attr));
    const int ncg = (p.maxcols * (int)nb + 7) / 8;
    const i64 grid = (p.items * ncg + PW - 1) / PW;
    k_pair_wmbej<FT><<<(unsigned)grid, PW * 32, pb_smem<FT>(), stream()>>>(
        p.d_groups, (int)p.groups.size(), p.items, ncg, V.arr, r.arr, W.arr, f, (int)nb, r.bs, wb);
    count_launch();
    return cuda_check(cudaGetLastError(), "k_pair_wmbej");
}

constexpr size_t PB_SMEM_MOST = 227 * 1024;

template <int FT>
int fae_go(const PairBlkPlan &p, const Ten &V, const Ten &r, Ten &F, double f, i64 nb, i64 fb) {
    static std::atomic<bool> attr{false};
    CPSD_TRY(pb_attr<FT>((const void *)k_pair_fae<FT>, PB_SMEM_MOST, attr));
    const size_t smem = pb_smem<FT>() + sizeof(double) * PW * 8 * (size_t)p.maxe;
    for (int c0 = 0; c0 < (int)nb; c0 += 8) {
        k_pair_fae<FT><<<(unsigned)p.nrow, PW * 32, smem, stream()>>>(p.d_groups, p.d_glist, p.d_rowirr, V.arr, r.arr,
                                                                      F.arr, f, c0, (int)nb, r.bs, fb, p.maxe);
        count_launch();
    }
    return cuda_check(cudaGetLastError(), "k_pair_fae");
}

}  // namespace

int PairBlkPlan::upload() {
    if (uploaded.load(std::memory_order_acquire)) return CPSD_OK;
    std::lock_guard<std::mutex> lock(upload_mutex());
    if (uploaded.load(std::memory_order_relaxed)) return CPSD_OK;
    CPSD_TRY(upload_table(groups, &d_groups, "pair plan"));
    CPSD_TRY(upload_table(glist, &d_glist, "pair plan"));
    CPSD_TRY(upload_table(rowirr, &d_rowirr, "pair plan"));
    // the tables may next be read by kernels on another thread's stream
    CPSD_TRY(cuda_check(cudaStreamSynchronize(stream()), "plan upload"));
    uploaded.store(true, std::memory_order_release);
    return CPSD_OK;
}

bool pairblk_wmbej_takes(const Ten &V, const Ten &r, const Ten &W, i64 nb) {
    const Desc &v = V.d, &s = r.d, &w = W.d;
    return layouts_ok(V, r) && w.sym == s.sym && w.iop[0] == 1 && w.iop[1] == 1 && same_pop(w.pop[0], v.pop[0]) &&
           same_pop(w.pop[1], v.pop[3]) && same_pop(w.pop[2], v.pop[2]) && same_pop(w.pop[3], s.pop[1]) &&
           !(nb > 1 && r.bs == 0);
}

bool pairblk_fae_takes(const Ten &V, const Ten &r, const Ten &F, i64 nb) {
    const Desc &v = V.d, &s = r.d, &w = F.d;
    return layouts_ok(V, r) && w.sym == s.sym && w.iop[0] == 1 && w.iop[1] == 1 && same_pop(w.pop[0], v.pop[0]) &&
           same_pop(w.pop[1], v.pop[0]) && is_zorb8(w.pop[2]) && is_zorb8(w.pop[3]) && !(nb > 1 && r.bs == 0);
}

int pairblk_wmbej(const Ten &V, const Ten &r, Ten &W, double f, i64 nb, double flops, bool *done) {
    *done = false;
    const Desc &v = V.d, &s = r.d, &w = W.d;
    static std::map<std::string, std::unique_ptr<PairBlkPlan>> cache;
    static std::mutex mx;
    PairBlkPlan *p;
    CPSD_TRY(cached(cache, mx, v.key() + s.key() + w.key() + sym_key(), &p, [&](PairBlkPlan &P) {
        const i64 n = ctx().nirrep;
        const i64 *pv = v.pop[0], *po = v.pop[3];
        for (i64 hx = 1; hx <= n; hx++)
            for (i64 hm = 1; hm <= n; hm++) {
                const i64 h = dp(hx, hm), nl = v.nleft(h);
                if (pv[hx - 1] == 0 || po[hm - 1] == 0 || nl == 0) continue;
                const i64 col = v.block_base(h) + (isymoffso(hm, h, v.pop[2], v.pop[3], 1) - 1) * nl;
                for (i64 hq = 1; hq <= n; hq++) {
                    const i64 hp = dp(hq, h);
                    if (hp > hq || pv[hp - 1] == 0 || pv[hq - 1] == 0) continue;
                    PairGroup g{};
                    g.np = (int)pv[hp - 1];
                    g.nq = (int)pv[hq - 1];
                    g.tri = hp == hq;
                    g.nx = (int)pv[hx - 1];
                    g.nm = (int)po[hm - 1];
                    g.v = col + pair_off(v, hq, h);
                    g.vx = nl;
                    g.vm = nl * pv[hx - 1];
                    // out(e; m, x, j) of the rows e of irrep he with the
                    // columns j of the irrep that r pairs with the other index
                    auto out = [&](i64 he, i64 hj, i64 *o, i64 *ox, i64 *om, i64 *oj) {
                        const i64 L = dp(he, hm), R = dp(hx, hj), nw = w.nleft(L);
                        *o = w.block_base(R) + (isymoffso(hj, R, w.pop[2], w.pop[3], 1) - 1) * nw +
                             isymoffso(hm, L, w.pop[0], w.pop[1], 1) - 1;
                        *ox = nw;
                        *om = pv[he - 1];
                        *oj = nw * pv[hx - 1];
                    };
                    const i64 jq = dp(hq, s.sym), jp = dp(hp, s.sym);
                    g.ncp = (int)po[jq - 1];
                    g.ncq = (int)po[jp - 1];
                    if (g.ncp) {
                        g.rq = vec_off(s, jq);
                        g.rqj = pv[hq - 1];
                        out(hp, jq, &g.op, &g.opx, &g.opm, &g.opj);
                    }
                    if (g.ncq) {
                        g.rp = vec_off(s, jp);
                        g.rpj = pv[hp - 1];
                        out(hq, jp, &g.oq, &g.oqx, &g.oqm, &g.oqj);
                    }
                    if (!g.ncp && !g.ncq) continue;
                    g.start = (int)P.items;
                    P.items += (i64)g.nx * g.nm;
                    P.maxp = std::max(P.maxp, g.np);
                    P.maxcols = std::max({P.maxcols, g.ncp, g.ncq});
                    P.groups.push_back(g);
                }
            }
    }));
    const i64 ncg = ((i64)p->maxcols * nb + 7) / 8;
    if (p->items * std::max<i64>(ncg, 1) > 0x7fffffffLL) return CPSD_OK;
    *done = true;
    if (p->groups.empty()) return CPSD_OK;
    CPSD_TRY(p->upload());
    cudaEvent_t end;
    CPSD_TRY(timing_begin(flops, (i64)p->groups.size(), p->items * ncg, W.len() * nb, 23, &end));
    const i64 wb = nb > 1 ? (W.bs ? W.bs : W.len()) : 0;
    // strips of 32 rows at every size: with 4, 8 and 12 row tiles of 8 the
    // launch took 22, 33, 39 us at 32 rows an irrep (C2v, 12 occupied), 55, 59,
    // 70 at 48, 88, 94, 115 at 64, 148, 172, 154 at 72, 254, 307, 258 at 96,
    // 336, 342, 404 at 97, 555, 549, 675 at 128; 72, 68, 74 at 160 without symmetry
    CPSD_TRY(wmbej_go<4>(*p, V, r, W, f, nb, wb));
    return timing_end(end);
}

int pairblk_fae(const Ten &V, const Ten &r, Ten &F, double f, i64 nb, double flops, bool *done) {
    *done = false;
    const Desc &v = V.d, &s = r.d, &w = F.d;
    static std::map<std::string, std::unique_ptr<PairBlkPlan>> cache;
    static std::mutex mx;
    PairBlkPlan *p;
    CPSD_TRY(cached(cache, mx, v.key() + s.key() + w.key() + sym_key(), &p, [&](PairBlkPlan &P) {
        const i64 n = ctx().nirrep;
        const i64 *pv = v.pop[0], *po = v.pop[3];
        for (i64 ha = 1; ha <= n; ha++) {
            P.glist.push_back((int)P.groups.size());
            const i64 he = dp(ha, s.sym);
            P.maxe = std::max(P.maxe, (int)pv[he - 1]);
            for (i64 a = 0; a < pv[ha - 1]; a++) {
                P.rowirr.push_back((int)ha - 1);
                P.rowirr.push_back((int)a);
                P.nrow++;
            }
            for (i64 hm = 1; hm <= n && pv[ha - 1] > 0; hm++) {
                const i64 h = dp(ha, hm), hf = dp(hm, s.sym), nl = v.nleft(h);
                if (po[hm - 1] == 0 || pv[hf - 1] == 0 || pv[he - 1] == 0) continue;
                const i64 hp = std::min(he, hf), hq = std::max(he, hf);
                PairGroup g{};
                g.np = (int)pv[hp - 1];
                g.nq = (int)pv[hq - 1];
                g.tri = hp == hq;
                g.nx = (int)pv[ha - 1];
                g.nm = (int)po[hm - 1];
                g.v = v.block_base(h) + (isymoffso(hm, h, v.pop[2], v.pop[3], 1) - 1) * nl + pair_off(v, hq, h);
                g.vx = nl;
                g.vm = nl * pv[ha - 1];
                // stored (e,f): sum over q = f with V; stored (f,e): sum over
                // p = f with -V
                g.ncp = he == hp;
                g.ncq = he == hq;
                g.rq = g.rp = vec_off(s, hm);
                g.rqm = g.rpm = pv[hf - 1];
                g.op = isymoffso(he, w.sym, w.pop[0], w.pop[1], 1) - 1;
                g.opx = 1;
                g.opj = pv[ha - 1];  // stride of e
                P.maxp = std::max(P.maxp, g.np);
                P.groups.push_back(g);
            }
        }
        P.glist.push_back((int)P.groups.size());
    }));
    if (pb_smem<8>() + sizeof(double) * PW * 8 * (size_t)p->maxe > PB_SMEM_MOST) return CPSD_OK;
    *done = true;
    if (p->groups.empty()) return CPSD_OK;
    CPSD_TRY(p->upload());
    cudaEvent_t end;
    CPSD_TRY(timing_begin(flops, (i64)p->groups.size(), p->nrow, F.len() * nb, 23, &end));
    const i64 fb = nb > 1 ? (F.bs ? F.bs : F.len()) : 0;
    // 4, 8 and 12 row tiles, us a launch: 18, 21, 27 at 32 rows an irrep (C2v),
    // 38, 35, 47 at 48, 51, 45, 59 at 64, 74, 74, 71 at 72, 115, 117, 119 at 96,
    // 150, 129, 180 at 97, 285, 279, 336 at 128; 94, 104, 109 at 160 without
    // symmetry.  Two instances come within a tenth of the best everywhere.
    if (p->maxp <= 32) CPSD_TRY(fae_go<4>(*p, V, r, F, f, nb, fb));
    else CPSD_TRY(fae_go<8>(*p, V, r, F, f, nb, fb));
    return timing_end(end);
}

}  // namespace cpsd
