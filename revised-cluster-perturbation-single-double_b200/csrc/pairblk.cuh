// Products of a packed antisymmetric pair with singles vectors, straight from
// the packed list: W(em,bj) += r(f,j) V(fe,bm), the singles update of the
// ring intermediate (Wmbej_r1abci), and F(a,e) += r(f,m) V(ef,am)
// (Fae_r1abci).  The general path expands the pair first, which doubles the
// list and writes and reads it once more.
#pragma once
#include <atomic>
#include <memory>
#include <string>

#include "ops.hpp"

namespace cpsd {

// One irrep block of the packed pair for the columns (x, m) of one irrep
// assignment: rows p < np, q < nq (p < q where tri), p fastest.  The block
// of column (x, m) starts at v + x vx + m vm.  Its two products are
//   out(p, c) += sp f sum_q V(p,q) r(q, c),  out(q, c) += sq f sum_p V(p,q) r(p, c)
// with r(q, c) at rq + q + col offset (j rqj + root batch) and out(p, c) at
// op + x ox + p os + j opj + ...; nc* = 0 where a side has no partner.
struct PairGroup {
    int start;  // first work item (task mode) or first group of a row's list
    int np, nq, tri, nx, nm;
    int ncp, ncq;  // columns j of the p and the q product (per root)
    i64 v, vx, vm;
    i64 rq, rqj, rqm;  // r of the p product: rows q
    i64 rp, rpj, rpm;  // r of the q product: rows p
    i64 op, opx, opm, opj;
    i64 oq, oqx, oqm, oqj;
};

struct PairBlkPlan {
    std::vector<PairGroup> groups;
    i64 items = 0;
    int maxp = 0;      // most rows p of a block
    int maxcols = 0;   // most columns of a product, all roots
    // F(a,e): groups of irrep h_a are glist[h_a] .. glist[h_a + 1]
    std::vector<int> glist;
    int nrow = 0, maxe = 0;
    std::atomic<bool> uploaded{false};
    PairGroup *d_groups = nullptr;
    int *d_glist = nullptr, *d_rowirr = nullptr;
    std::vector<int> rowirr;  // irrep and index in it of every row a
    int upload();
};

// whether the layouts are those of a packed (vv|vo) list, a singles vector and a
// full (vo|vo) result, or (vv) result; the calls below take no others
bool pairblk_wmbej_takes(const Ten &V, const Ten &r, const Ten &W, i64 nb);
bool pairblk_fae_takes(const Ten &V, const Ten &r, const Ten &F, i64 nb);
// W(em,bj) += f r(f,j) V(fe,bm) for nb roots; *done = false (and nothing
// queued) when the sizes are beyond the kernel's.  flops: of the contraction,
// for the timing record
int pairblk_wmbej(const Ten &V, const Ten &r, Ten &W, double f, i64 nb, double flops, bool *done);
// F(a,e) += f r(f,m) V(ef,am)
int pairblk_fae(const Ten &V, const Ten &r, Ten &F, double f, i64 nb, double flops, bool *done);

}  // namespace cpsd
