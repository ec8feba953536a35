// Execution plan of the GPU numeric phase (see plan.h).
#include "plan.h"
#include "smhash.h"

#include <thread>

#include <algorithm>
#include <cmath>
#include <map>

namespace sprb {

namespace {

// First-fit allocator over a linear arena, in units of doubles.  Blocks are
// aligned to 32 doubles (256 bytes) so every front starts on a TMA/vector
// friendly boundary.
class Arena {
public:
    int64_t alloc(int64_t n) {
        n = (n + 31) / 32 * 32;
        if (n == 0) n = 32;
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            if (it->second >= n) {
                int64_t off = it->first;
                int64_t rest = it->second - n;
                free_.erase(it);
                if (rest > 0) free_[off + n] = rest;
                return off;
            }
        }
        int64_t off = top_;
        top_ += n;
        peak_ = std::max(peak_, top_);
        return off;
    }
    void release(int64_t off, int64_t n) {
        n = (n + 31) / 32 * 32;
        if (n == 0) n = 32;
        auto it = free_.emplace(off, n).first;
        // coalesce with the next block
        auto nx = std::next(it);
        if (nx != free_.end() && it->first + it->second == nx->first) {
            it->second += nx->second;
            free_.erase(nx);
        }
        // coalesce with the previous block
        if (it != free_.begin()) {
            auto pv = std::prev(it);
            if (pv->first + pv->second == it->first) {
                pv->second += it->second;
                free_.erase(it);
                it = pv;
            }
        }
        // shrink the top
        if (it->first + it->second == top_) {
            top_ = it->first;
            free_.erase(it);
        }
    }
    int64_t peak() const { return peak_; }

private:
    std::map<int64_t, int64_t> free_;
    int64_t top_ = 0;
    int64_t peak_ = 0;
};

inline int32_t round_up4(int32_t x) { return (x + 3) / 4 * 4; }

}  // namespace

int build_plan(const int64_t* mspar, const int64_t* mtrees, const int64_t* msifa, Plan& P) {
    // Pointer conventions of SPRFC1 (src/SPR/sprfc1.f:165-196).
    P.neq = mspar[7];
    P.nsuper = mspar[10];
    P.maxsup = mspar[12];
    P.mfront = mspar[13];
    P.nofsub = mspar[14];
    P.nzerol = mspar[15];
    const int64_t ns = P.nsuper;
    if (ns <= 0 || P.neq <= 0 || mspar[44] < 1 || mspar[45] < 1 || mspar[46] < 1 || mspar[47] < 1)
        return -2;
    const int64_t* xsuper = mtrees + (mspar[44] - 1);
    const int64_t* xsibl = xsuper + (ns + 1);
    const int64_t* sibl = xsuper + 2 * (ns + 1);
    const int64_t* xlindx = mtrees + (mspar[45] - 1);
    const int64_t* lindx = msifa + (mspar[46] - 1);
    const int64_t* xlnz = msifa + (mspar[47] - 1);
    const int64_t* supsup = xlindx + (ns + 1);          // sprfc1.f:183
    const bool lpar57 = mspar[56] > 0;

    P.retained.assign(ns, 0);
    P.any_retained = false;
    if (lpar57)
        for (int64_t js = 0; js < ns; ++js)
            if (supsup[js] > 0) {
                P.retained[js] = 1;
                P.any_retained = true;
            }
    P.fst.resize(ns);
    P.S.resize(ns);
    P.F.resize(ns);
    P.parent.assign(ns, -1);
    P.level.assign(ns, 0);
    P.lnz_off.resize(ns);
    P.lindx_off.resize(ns);
    P.child_ptr.assign(ns + 1, 0);
    P.factor_flops = 0.0;
    P.solve_flops = 0.0;
    for (int64_t js = 0; js < ns; ++js) {
        P.fst[js] = (int32_t)(xsuper[js] - 1);
        P.S[js] = (int32_t)(xsuper[js + 1] - xsuper[js]);
        P.F[js] = (int32_t)(xlindx[js + 1] - xlindx[js]);
        P.lnz_off[js] = xlnz[js] - 1;
        P.lindx_off[js] = xlindx[js] - 1;
        if (P.S[js] <= 0 || P.F[js] < P.S[js]) return -2;
        if (P.retained[js]) continue;                  // sprtrs.f:1956
        const double s = P.S[js], f = P.F[js];
        // RINFO(3) and RINFO(4) per supernode, src/SPR/sprtrs.f:1961-1980
        P.factor_flops += ((f * f) + 2.0 * f) * s - 2.0 * (1.0 + f) * (s * (s + 1.0) / 2.0) +
                          s * (s + 1.0) * (2.0 * s + 1.0) / 6.0;
        P.solve_flops += f * s - s * (s - 1.0) / 2.0 - s;
    }
    P.solve_flops = 2.0 * P.solve_flops + (double)P.neq;
    // children (SIBL order) and parents
    P.child.clear();
    for (int64_t js = 0; js < ns; ++js) {
        P.child_ptr[js] = (int32_t)P.child.size();
        for (int64_t k = xsibl[js]; k < xsibl[js + 1]; ++k) {
            int64_t c = sibl[k - 1] - 1;
            if (c < 0 || c >= js) return -2;   // postorder: children precede parents
            P.child.push_back((int32_t)c);
            P.parent[c] = (int32_t)js;
        }
    }
    P.child_ptr[ns] = (int32_t)P.child.size();
    // rows (0-based)
    P.rows.resize(xlindx[ns] - 1);
    for (size_t i = 0; i < P.rows.size(); ++i) P.rows[i] = (int32_t)(lindx[i] - 1);
    // levels: leaves 0, parent = 1 + max(children)
    int32_t nlev = 0;
    for (int64_t js = 0; js < ns; ++js) {
        int32_t lv = 0;
        for (int32_t k = P.child_ptr[js]; k < P.child_ptr[js + 1]; ++k)
            lv = std::max(lv, P.level[P.child[k]] + 1);
        P.level[js] = lv;
        nlev = std::max(nlev, lv + 1);
    }
    // relative maps (SPRF12 merge) and the contribution lists
    P.rel_off.assign(ns, -1);
    P.rel.clear();
    P.rbase.assign(ns + 1, 0);
    for (int64_t js = 0; js < ns; ++js) P.rbase[js + 1] = P.rbase[js] + P.F[js];
    std::vector<int64_t> ccount(P.rbase[ns] + 1, 0);
    for (int64_t c = 0; c < ns; ++c) {
        const int32_t q = P.F[c] - P.S[c];
        const int32_t p = P.parent[c];
        if (q <= 0) continue;
        if (p < 0) return -2;                  // update rows without a parent
        P.rel_off[c] = (int64_t)P.rel.size();
        const int32_t* prow = &P.rows[P.lindx_off[p]];
        const int32_t* crow = &P.rows[P.lindx_off[c] + P.S[c]];
        int32_t sup = 0;
        for (int32_t t = 0; t < q; ++t) {
            while (sup < P.F[p] && prow[sup] < crow[t]) ++sup;
            if (sup >= P.F[p] || prow[sup] != crow[t]) return -4;   // not a subset
            P.rel.push_back(sup);
            ccount[P.rbase[p] + sup + 1]++;
            ++sup;
        }
    }
    P.cptr.assign(P.rbase[ns] + 1, 0);
    for (int64_t i = 0; i < P.rbase[ns]; ++i) P.cptr[i + 1] = P.cptr[i] + ccount[i + 1];
    P.cchild.assign(P.cptr[P.rbase[ns]], 0);
    P.ct.assign(P.cptr[P.rbase[ns]], 0);
    {
        std::vector<int64_t> fill(P.cptr.begin(), P.cptr.end() - 1);
        // children in the reference's assembly order: last sibling first (sprfc1.f:534)
        for (int64_t p = 0; p < ns; ++p) {
            for (int32_t k = P.child_ptr[p + 1] - 1; k >= P.child_ptr[p]; --k) {
                const int32_t c = P.child[k];
                const int32_t q = P.F[c] - P.S[c];
                for (int32_t t = 0; t < q; ++t) {
                    const int32_t j = P.rel[P.rel_off[c] + t];
                    const int64_t pos = fill[P.rbase[p] + j]++;
                    P.cchild[pos] = c;
                    P.ct[pos] = t;
                }
            }
        }
    }
    // arena layout, level by level
    P.buf_off.assign(ns, 0);
    P.buf_ld.assign(ns, 0);
    P.upd_off.assign(ns, 0);
    P.levels.assign(nlev, LevelPlan());
    std::vector<std::vector<int32_t>> bylev(nlev);
    for (int64_t js = 0; js < ns; ++js) bylev[P.level[js]].push_back((int32_t)js);
    std::vector<int64_t> buf_size(ns, 0);
    Arena arena;
    P.any_large = false;
    for (int32_t L = 0; L < nlev; ++L) {
        LevelPlan& lp = P.levels[L];
        std::vector<int32_t> nodes = bylev[L];
        // big buffers first: less fragmentation
        std::stable_sort(nodes.begin(), nodes.end(),
                         [&](int32_t a, int32_t b) { return P.F[a] > P.F[b]; });
        for (int32_t js : nodes) {
            const int32_t f = P.F[js], s = P.S[js], q = f - s;
            if (f <= kSmallMaxF) {
                lp.small_nodes.push_back(js);
                lp.small_maxF = std::max(lp.small_maxF, f);
                P.buf_ld[js] = std::max(q, 1);
                buf_size[js] = (int64_t)q * q;
                P.buf_off[js] = arena.alloc(buf_size[js]);
                P.upd_off[js] = P.buf_off[js];
            } else {
                lp.large_nodes.push_back(js);
                P.any_large = true;
                const int32_t ld = round_up4(f);
                P.buf_ld[js] = ld;
                buf_size[js] = (int64_t)ld * f;
                P.buf_off[js] = arena.alloc(buf_size[js]);
                P.upd_off[js] = P.buf_off[js] + (int64_t)s * ld + s;
            }
        }
        // small_nodes are in decreasing F: cut them into size classes
        {
            auto cls = [](int32_t f) { return f <= 64 ? 0 : f <= 96 ? 1 : f <= 128 ? 2 : 3; };
            for (int32_t k = 0; k < (int32_t)lp.small_nodes.size();) {
                const int32_t c = cls(P.F[lp.small_nodes[k]]);
                int32_t e = k;
                while (e < (int32_t)lp.small_nodes.size() && cls(P.F[lp.small_nodes[e]]) == c) ++e;
                int32_t nl = 0;
                for (int32_t q = k; q < e; ++q) {
                    const int32_t f = P.F[lp.small_nodes[q]], w = P.S[lp.small_nodes[q]];
                    nl = std::max(nl, f * w - w * (w - 1) / 2);
                }
                lp.small_classes.push_back(LevelPlan::SmallClass{k, e - k, P.F[lp.small_nodes[k]], nl});
                k = e;
            }
        }
        // after this level is assembled, its children are no longer needed
        for (int32_t js : nodes)
            for (int32_t k = P.child_ptr[js]; k < P.child_ptr[js + 1]; ++k) {
                const int32_t c = P.child[k];
                arena.release(P.buf_off[c], buf_size[c]);
            }
    }
    P.arena_doubles = arena.peak();
    P.linv_off.assign(ns, -1);
    P.linv_doubles = 0;
    for (int64_t js = 0; js < ns; ++js)
        if (P.F[js] > kSmallMaxF) {
            P.linv_off[js] = P.linv_doubles;
            P.linv_doubles += (int64_t)((P.S[js] + kNB - 1) / kNB) * kNB * kNB;
        }
    // ---- batched launches of the large path
    P.jobs.clear();
    P.alt.clear();
    P.rect_off.assign(ns, 0);
    P.rect_entries = 0;
    P.fwd_off.assign(ns, 0);
    P.fwd_entries = 0;
    auto open_launch = [&](Launch& l) { l.job_begin = (int64_t)P.jobs.size(); l.ntasks = 0; };
    auto add_job = [&](Launch& l, Job j, int64_t ntask, bool keep_empty = false) {
        if (ntask <= 0 && !keep_empty) return;
        j.task0 = l.ntasks;
        P.jobs.push_back(j);
        l.ntasks += std::max<int64_t>(ntask, 0);
    };
    auto close_launch = [&](Launch& l) { l.job_count = (int64_t)P.jobs.size() - l.job_begin; };
    P.gemm_flops = 0.0;
    P.tc_flops = 0.0;
    P.slab_rows = 0;
    P.slab_rows_far = 0;
    P.i8_rows = P.i8_scales = 0;
    P.small_flops = 0.0;
    for (int64_t js = 0; js < ns; ++js)
        if (P.F[js] <= kSmallMaxF) {
            const double s = P.S[js], f = P.F[js];
            P.small_flops += ((f * f) + 2.0 * f) * s - 2.0 * (1.0 + f) * (s * (s + 1.0) / 2.0) +
                             s * (s + 1.0) * (2.0 * s + 1.0) / 6.0;
        }
    // lower-triangle entries of rows [c0, r_end) x columns [c0, c_end), times 2K
    auto update_flops = [](int32_t c0, int32_t c_end, int32_t r_end, int32_t k) -> double {
        double e = 0.0;
        const double n = c_end - c0, r = r_end - c0;
        e = n * r - n * (n - 1.0) / 2.0;
        return 2.0 * e * k;
    };
    auto tiles_t = [](int32_t c0, int32_t c_end, int32_t r_end, int32_t t) -> int64_t {
        const int64_t nct = (c_end - c0 + t - 1) / t;
        const int64_t nr = (r_end - c0 + t - 1) / t;
        return nct * nr - nct * (nct - 1) / 2;
    };
    for (int32_t L = 0; L < nlev; ++L) {
        LevelPlan& lp = P.levels[L];
        if (lp.large_nodes.empty()) continue;
        open_launch(lp.assemble);
        for (int32_t js : lp.large_nodes)
            add_job(lp.assemble, Job{js, 0, P.F[js], P.F[js], 0, 0, 0}, P.F[js]);
        close_launch(lp.assemble);
        // elimination, Schur updates and the solve steps: retained fronts excluded
        lp.elim_nodes.clear();
        for (int32_t js : lp.large_nodes)
            if (!P.retained[js]) lp.elim_nodes.push_back(js);
        const std::vector<int32_t>& elim = lp.elim_nodes;
        int32_t smax = 0;
        for (int32_t js : elim) smax = std::max(smax, P.S[js]);
        const int32_t nsteps = (smax + kNB - 1) / kNB;
        lp.panel.assign(nsteps, Launch());
        lp.update.assign(nsteps, std::vector<Launch>());
        // Schur-update jobs of one step, split into a big-tile and a small-tile launch
        auto emit_updates = [&](std::vector<Job>& jl, std::vector<Launch>& out) {
            for (int pass = 0; pass < 2; ++pass) {
                const int32_t tile = pass == 0 ? kTileBig : kTile;
                Launch l;
                l.tile = tile;
                open_launch(l);
                for (const Job& j : jl) {
                    const bool big = (j.r_end - j.c0) >= 4 * kTileBig;
                    if (big != (pass == 0)) continue;
                    add_job(l, j, tiles_t(j.c0, j.c_end, j.r_end, tile));
                }
                close_launch(l);
                l.tile = tile;
                if (l.ntasks <= 0) continue;
                if (pass == 1) {
                    // the same jobs in kTileTiny tiles, for the tile autotuner
                    Launch a;
                    open_launch(a);
                    for (const Job& j : jl)
                        if ((j.r_end - j.c0) < 4 * kTileBig) add_job(a, j, tiles_t(j.c0, j.c_end, j.r_end, kTileTiny));
                    close_launch(a);
                    a.tile = kTileTiny;
                    l.alt = (int32_t)P.alt.size();
                    P.alt.push_back(a);
                }
                out.push_back(l);
            }
        };
        // the far and K = S updates for the tensor-core path: slabs of W = L D
        // and L as FP32 hi/lo pairs (4 arrays of K blocks of [rows][32])
        auto emit_tc = [&](std::vector<Job> jl, std::vector<TcLaunch>& out, int64_t& slab_max) {
            if (jl.empty()) return;
            int64_t rows = 0;
            for (Job& j : jl) {
                const int64_t np = (int64_t)(j.r_end - j.c0 + kTcTile - 1) / kTcTile * kTcTile;
                const int64_t nkb = (j.k_hi - j.k_lo + kTcBK - 1) / kTcBK;
                j.slab = rows;
                rows += 4 * nkb * np;
            }
            TcLaunch t;
            open_launch(t.split);
            for (const Job& j : jl) {
                const int64_t np = (int64_t)(j.r_end - j.c0 + kTcTile - 1) / kTcTile * kTcTile;
                const int64_t nkb = (j.k_hi - j.k_lo + kTcBK - 1) / kTcBK;
                add_job(t.split, j, (np / 32) * nkb);
            }
            close_launch(t.split);
            open_launch(t.gemm);
            for (const Job& j : jl) add_job(t.gemm, j, tiles_t(j.c0, j.c_end, j.r_end, kTcTile));
            close_launch(t.gemm);
            t.gemm.tile = kTcTile;
            slab_max = std::max(slab_max, rows);
            out.push_back(t);
        };
        // an integer-digit update: jobs jl (and the far part of the same panels,
        // jfar, whose first column lies a multiple of kI8TileM after its job's)
        auto emit_i8 = [&](const std::vector<Job>& jl, const std::vector<Job>& jfar, I8Launch& out) {
            int64_t rows = 0, sc = 0;
            std::vector<Job> base, small, small_far;
            for (const Job& j : jl)
                (j.r_end - j.c0 >= kI8MinRows && j.k_hi - j.k_lo >= kI8MinK ? base : small).push_back(j);
            for (const Job& j : jfar)
                for (const Job& k : small)
                    if (k.node == j.node) small_far.push_back(j);
            emit_updates(small, out.rest);
            emit_updates(small_far, out.far_rest);
            if (base.empty()) return;
            for (const Job& j : base) out.flops += update_flops(j.c0, j.c_end, j.r_end, j.k_hi - j.k_lo);
            for (Job& j : base) {
                const int64_t nkb = (j.k_hi - j.k_lo + kI8BK - 1) / kI8BK;
                j.np = (int32_t)((j.r_end - j.c0 + kI8TileM - 1) / kI8TileM * kI8TileM);
                j.slab = rows;
                j.aux_job = sc;
                j.aux = sc + 8;
                rows += 2 * nkb * kI8Digits * j.np;
                sc += 8 + j.np;
            }
            P.i8_rows = std::max(P.i8_rows, rows);
            P.i8_scales = std::max(P.i8_scales, sc);
            auto tiles = [](const Job& j) -> int64_t {
                const int64_t nct = (j.c_end - j.c0 + kI8TileN - 1) / kI8TileN;
                const int64_t nr = (j.r_end - j.c0 + kI8TileM - 1) / kI8TileM;
                int64_t n = 0;
                for (int64_t it = 0; it < nr; ++it) n += std::min(nct, 2 * it + 2);
                return n;
            };
            open_launch(out.split);
            for (const Job& j : base) add_job(out.split, j, j.np / 32);
            close_launch(out.split);
            open_launch(out.gemm);
            for (const Job& j : base) add_job(out.gemm, j, tiles(j));
            close_launch(out.gemm);
            open_launch(out.far);
            for (const Job& f : jfar)
                for (const Job& b : base)
                    if (b.node == f.node) {
                        Job j = f;
                        j.np = b.np;
                        j.slab = b.slab + (f.c0 - b.c0);
                        j.aux_job = b.aux_job;
                        j.aux = b.aux + (f.c0 - b.c0);
                        out.flops += update_flops(j.c0, j.c_end, j.r_end, j.k_hi - j.k_lo);
                        add_job(out.far, j, tiles(j));
                    }
            close_launch(out.far);
            out.gemm.tile = out.far.tile = kI8TileM;
        };
        lp.trail_i8.assign(nsteps, I8Launch());
        lp.outer_i8.clear();
        lp.far.assign(nsteps, std::vector<Launch>());
        lp.ahead.assign(nsteps, std::vector<Launch>());
        lp.next_tc.assign(nsteps, std::vector<TcLaunch>());
        lp.next_flops.assign(nsteps, 0.0);
        lp.far_tc.assign(nsteps, std::vector<TcLaunch>());
        lp.far_flops.assign(nsteps, 0.0);
        for (int32_t st = 0; st < nsteps; ++st) {
            const int32_t k0 = st * kNB;
            open_launch(lp.panel[st]);
            for (int32_t js : elim) {
                const int32_t s = P.S[js], f = P.F[js];
                if (k0 >= s) continue;
                const int32_t nb = std::min(kNB, s - k0);
                const int64_t nrb = (f - (k0 + nb) + kTRSMRows - 1) / kTRSMRows;
                add_job(lp.panel[st], Job{js, k0 + nb, k0 + nb, f, k0, k0 + nb, 0}, nrb, true);
            }
            close_launch(lp.panel[st]);
            std::vector<Job> jl, jahead, jfar;
            for (int32_t js : elim) {
                const int32_t s = P.S[js], f = P.F[js];
                if (k0 >= s) continue;
                const int32_t nb = std::min(kNB, s - k0);
                const int32_t c0 = k0 + nb;
                const int32_t sp0 = (k0 / kSuperPanel) * kSuperPanel;
                const int32_t sp1 = std::min(sp0 + kSuperPanel, s);
                if (c0 < sp1) {                                     // inside the super-panel
                    // the next panel's columns with the panel's own launch (by
                    // this panel and the one before), the ones after the next
                    // two panels beside the next step
                    const int32_t c2 = c0 + 2 * kNB;
                    if (c2 < sp1) {
                        jahead.push_back(Job{js, c2, sp1, f, k0, c0, 0});
                        P.gemm_flops += update_flops(c2, sp1, f, nb);
                    }
                }
                if (c0 == sp1 && sp1 < s) {                          // trailing, K = kSuperPanel
                    // the next super-panel's columns now; the columns beyond
                    // it on the side stream, overlapping that super-panel
                    const int32_t sp2 = std::min(sp1 + kSuperPanel, s);
                    jl.push_back(Job{js, sp1, sp2, f, sp0, sp1, 0});
                    P.gemm_flops += update_flops(sp1, sp2, f, sp1 - sp0);
                    lp.next_flops[st] += update_flops(sp1, sp2, f, sp1 - sp0);
                    if (sp2 < s) {
                        jfar.push_back(Job{js, sp2, s, f, sp0, sp1, 0});
                        P.gemm_flops += update_flops(sp2, s, f, sp1 - sp0);
                        P.tc_flops += update_flops(sp2, s, f, sp1 - sp0);
                        lp.far_flops[st] += update_flops(sp2, s, f, sp1 - sp0);
                    }
                }
            }
            emit_updates(jl, lp.update[st]);
            if (lp.next_flops[st] > 0.0) {
                emit_tc(jl, lp.next_tc[st], P.slab_rows);
                emit_i8(jl, jfar, lp.trail_i8[st]);
            }
            emit_updates(jahead, lp.ahead[st]);
            emit_updates(jfar, lp.far[st]);
            emit_tc(jfar, lp.far_tc[st], P.slab_rows_far);
        }
        open_launch(lp.rect);
        int64_t roff = 0, foff = 0;
        for (int32_t js : elim) {
            const int32_t s = P.S[js], f = P.F[js];
            if (f <= s) continue;
            const int64_t nrc = (f - s + fwd_rows(s) - 1) / fwd_rows(s), ncc = (s + kFwdCols - 1) / kFwdCols;
            P.fwd_off[js] = foff;
            foff += ncc * (f - s);
            add_job(lp.rect, Job{js, 0, s, f, (int32_t)nrc, (int32_t)ncc, 0}, nrc * ncc);
        }
        close_launch(lp.rect);
        open_launch(lp.rect_back);
        for (int32_t js : elim) {
            const int32_t s = P.S[js], f = P.F[js];
            if (f <= s) continue;
            const int64_t nrc = (f - s + kRectRows - 1) / kRectRows, ncc = (s + kRectCols - 1) / kRectCols;
            P.rect_off[js] = roff;
            roff += nrc * s;
            add_job(lp.rect_back, Job{js, 0, s, f, (int32_t)nrc, (int32_t)ncc, 0}, nrc * ncc);
        }
        close_launch(lp.rect_back);
        P.rect_entries = std::max(P.rect_entries, roff);
        P.fwd_entries = std::max(P.fwd_entries, foff);
        open_launch(lp.rect_rows);
        for (int32_t js : elim) {
            const int32_t s = P.S[js], f = P.F[js];
            if (f > s && s > kFwdCols) add_job(lp.rect_rows, Job{js, s, f, f, 0, 0, 0}, f - s);
        }
        close_launch(lp.rect_rows);
        lp.retained_large = elim.size() != lp.large_nodes.size();
        {
            std::vector<Job> jl;
            for (int32_t js : elim) {
                const int32_t s = P.S[js], f = P.F[js];
                if (f > s) {
                    jl.push_back(Job{js, s, f, f, 0, s, 0});
                    P.gemm_flops += update_flops(s, f, f, s);
                    P.tc_flops += update_flops(s, f, f, s);
                    lp.outer_flops += update_flops(s, f, f, s);
                }
            }
            lp.outer.clear();
            emit_updates(jl, lp.outer);
            lp.outer_tc.clear();
            emit_tc(jl, lp.outer_tc, P.slab_rows);
            for (int32_t k0 = 0;; k0 += kI8MaxK) {
                std::vector<Job> jk;
                for (Job j : jl)
                    if (j.k_hi > k0) {
                        j.k_lo = k0;
                        j.k_hi = std::min(j.k_hi, k0 + kI8MaxK);
                        jk.push_back(j);
                    }
                if (jk.empty()) break;
                I8Launch t;
                emit_i8(jk, {}, t);
                if (k0 == 0 && t.gemm.ntasks <= 0) break;     // later parts have fewer jobs and columns
                lp.outer_i8.push_back(t);
            }
        }
        open_launch(lp.writeback);
        for (int32_t js : lp.large_nodes)
            add_job(lp.writeback, Job{js, 0, P.S[js], P.F[js], 0, 0, 0}, P.S[js]);
        close_launch(lp.writeback);
        const int32_t nst = (int32_t)lp.panel.size();
        lp.wb_sp.assign(nst, Launch());
        for (int32_t st = 0; st < nst; ++st) {
            open_launch(lp.wb_sp[st]);
            for (int32_t js : lp.elim_nodes) {
                const int32_t s = P.S[js], k0 = st * kNB;
                if (k0 >= s) continue;
                const int32_t k1 = std::min(k0 + kNB, s);
                if (k1 % kSuperPanel != 0 && k1 != s) continue;     // the step does not end a super-panel
                const int32_t sp0 = (k0 / kSuperPanel) * kSuperPanel;
                add_job(lp.wb_sp[st], Job{js, sp0, k1, P.F[js], 0, 0, 0}, k1 - sp0);
            }
            close_launch(lp.wb_sp[st]);
        }
    }
    // task -> job maps of every launch
    P.task_map.clear();
    auto build_map = [&](Launch& l) {
        l.map_begin = (int64_t)P.task_map.size();
        for (int64_t j = 0; j < l.job_count; ++j) {
            const int64_t t0 = P.jobs[l.job_begin + j].task0;
            const int64_t t1 = (j + 1 < l.job_count) ? P.jobs[l.job_begin + j + 1].task0 : l.ntasks;
            for (int64_t t = t0; t < t1; ++t) P.task_map.push_back((int32_t)j);
        }
    };
    for (Launch& l : P.alt) build_map(l);
    for (LevelPlan& lp : P.levels) {
        build_map(lp.assemble);
        build_map(lp.writeback);
        for (Launch& l : lp.wb_sp) build_map(l);
        build_map(lp.rect);
        build_map(lp.rect_back);
        build_map(lp.rect_rows);
        for (Launch& l : lp.panel) build_map(l);
        for (auto& v : lp.update)
            for (Launch& l : v) build_map(l);
        for (auto& v : lp.ahead)
            for (Launch& l : v) build_map(l);
        for (Launch& l : lp.outer) build_map(l);
        for (auto& v : lp.far)
            for (Launch& l : v) build_map(l);
        for (auto& v : lp.far_tc)
            for (TcLaunch& t : v) {
                build_map(t.split);
                build_map(t.gemm);
            }
        for (auto& v : lp.next_tc)
            for (TcLaunch& t : v) {
                build_map(t.split);
                build_map(t.gemm);
            }
        for (TcLaunch& t : lp.outer_tc) {
            build_map(t.split);
            build_map(t.gemm);
        }
        for (std::vector<I8Launch>* v : {&lp.trail_i8, &lp.outer_i8})
            for (I8Launch& t : *v) {
                build_map(t.split);
                build_map(t.gemm);
                build_map(t.far);
                for (Launch& l : t.rest) build_map(l);
                for (Launch& l : t.far_rest) build_map(l);
            }
    }
    // triangle tasks of the solves: per level, block-major (every task's
    // dependencies, the lower blocks of its own front, come earlier)
    P.tri_tasks.clear();
    for (LevelPlan& lp : P.levels) {
        std::vector<int32_t> fr;
        int32_t nbmax = 0;
        for (int32_t js : lp.elim_nodes) {
            if (P.F[js] <= kSmallMaxF) continue;
            fr.push_back(js);
            nbmax = std::max(nbmax, (P.S[js] + kNB - 1) / kNB);
        }
        lp.tri_begin = (int64_t)P.tri_tasks.size() / 2;
        for (int32_t b = 0; b < nbmax; ++b)
            for (int32_t js : fr)
                if (b * kNB < P.S[js]) {
                    P.tri_tasks.push_back(js);
                    P.tri_tasks.push_back(b);
                }
        lp.tri_count = (int64_t)P.tri_tasks.size() / 2 - lp.tri_begin;
    }
    return 0;
}

int64_t buffer_doubles(const Plan& P, int64_t js) {
    const int64_t f = P.F[js], s = P.S[js];
    return (f <= kSmallMaxF) ? (f - s) * (f - s) : (int64_t)P.buf_ld[js] * f;
}

// Every buffer inside the arena, and no two buffers that are live at the same
// level (from the node's own level to its parent's) overlap.
void check_plan(const Plan& P, int64_t& oob, int64_t& overlaps) {
    oob = 0;
    overlaps = 0;
    const int64_t ns = P.nsuper;
    for (int64_t js = 0; js < ns; ++js)
        if (P.buf_off[js] < 0 || P.buf_off[js] + buffer_doubles(P, js) > P.arena_doubles) ++oob;
    // index maps: a child's relative rows (SPRF12's LINDEX) lie in [0, F_p)
    // of its parent's rows, strictly increasing, and its column t lands in
    // parent column rel[t] exactly once in the contribution lists
    std::vector<int64_t> seen(P.rel.size(), 0);
    for (int64_t c = 0; c < ns; ++c) {
        const int32_t q = P.F[c] - P.S[c];
        if (q <= 0) continue;
        const int32_t p = P.parent[c];
        if (p < 0 || P.rel_off[c] < 0 || P.rel_off[c] + q > (int64_t)P.rel.size()) {
            ++oob;
            continue;
        }
        for (int32_t t = 0; t < q; ++t) {
            const int32_t r = P.rel[P.rel_off[c] + t];
            if (r < 0 || r >= P.F[p] || (t > 0 && r <= P.rel[P.rel_off[c] + t - 1])) ++oob;
        }
    }
    for (int64_t p = 0; p < ns; ++p)
        for (int32_t j = 0; j < P.F[p]; ++j)
            for (int64_t e = P.cptr[P.rbase[p] + j]; e < P.cptr[P.rbase[p] + j + 1]; ++e) {
                const int32_t c = P.cchild[e], t = P.ct[e];
                if (c < 0 || c >= ns || P.parent[c] != p || t < 0 || t >= P.F[c] - P.S[c] ||
                    P.rel[P.rel_off[c] + t] != j) {
                    ++oob;
                    continue;
                }
                ++seen[P.rel_off[c] + t];
            }
    for (int64_t k = 0; k < (int64_t)seen.size(); ++k)
        if (seen[k] != 1) ++oob;
    const int32_t nlev = (int32_t)P.levels.size();
    std::vector<std::vector<int32_t>> live(nlev);
    for (int64_t js = 0; js < ns; ++js) {
        const int32_t l0 = P.level[js];
        const int32_t l1 = P.parent[js] >= 0 ? P.level[P.parent[js]] : l0;
        for (int32_t L = l0; L <= l1; ++L) live[L].push_back((int32_t)js);
    }
    for (int32_t L = 0; L < nlev; ++L) {
        std::vector<std::pair<int64_t, int64_t>> iv;
        for (int32_t js : live[L]) {
            const int64_t n = buffer_doubles(P, js);
            if (n > 0) iv.emplace_back(P.buf_off[js], P.buf_off[js] + n);
        }
        std::sort(iv.begin(), iv.end());
        for (size_t k = 1; k < iv.size(); ++k)
            if (iv[k].first < iv[k - 1].second) ++overlaps;
    }
}

// the update that a panel step's launch makes of the next panel's columns, by
// its own panel and the one before it in the super-panel (empty past the last)
static Job chain_update(const Plan& P, const Job& panel) {
    Job j = panel;
    const int32_t sp0 = panel.k_lo / kSuperPanel * kSuperPanel;
    j.c0 = panel.k_hi;
    j.c_end = std::max(j.c0, std::min({j.c0 + kNB, sp0 + kSuperPanel, P.S[j.node]}));
    j.r_end = P.F[j.node];
    j.k_lo = std::max(sp0, panel.k_lo - kNB);
    return j;
}

void check_coverage(const Plan& P, int64_t& fp64, int64_t& tc) {
    fp64 = tc = 0;
    const int64_t ns = P.nsuper;
    for (int which = 0; which < 3; ++which) {          // 2: the FP64 lists with the integer-digit updates
        // per front: per column, the K intervals it receives
        std::vector<std::vector<std::vector<std::pair<int32_t, int32_t>>>> cov(ns);
        auto add = [&](const Launch& l) {
            for (int64_t j = 0; j < l.job_count; ++j) {
                const Job& jb = P.jobs[l.job_begin + j];
                auto& c = cov[jb.node];
                if (c.empty()) c.resize(P.F[jb.node]);
                for (int32_t col = jb.c0; col < jb.c_end; ++col) c[col].emplace_back(jb.k_lo, jb.k_hi);
            }
        };
        for (const LevelPlan& lp : P.levels) {
            for (size_t st = 0; st < lp.update.size(); ++st) {
                if (which == 2 && lp.trail_i8[st].gemm.ntasks > 0) {
                    add(lp.trail_i8[st].gemm);
                    add(lp.trail_i8[st].far);
                    for (const Launch& l : lp.trail_i8[st].rest) add(l);
                    for (const Launch& l : lp.trail_i8[st].far_rest) add(l);
                    continue;
                }
                for (const Launch& l : lp.update[st]) add(l);
            }
            for (const Launch& l : lp.panel)
                for (int64_t j = 0; j < l.job_count; ++j) {
                    const Job c = chain_update(P, P.jobs[l.job_begin + j]);
                    auto& v = cov[c.node];
                    if (v.empty()) v.resize(P.F[c.node]);
                    for (int32_t col = c.c0; col < c.c_end; ++col) v[col].emplace_back(c.k_lo, c.k_hi);
                }
            for (const auto& v : lp.ahead)
                for (const Launch& l : v) add(l);
            if (which == 0) {
                for (const auto& v : lp.far)
                    for (const Launch& l : v) add(l);
                for (const Launch& l : lp.outer) add(l);
            } else if (which == 2) {
                for (size_t st = 0; st < lp.far.size(); ++st)
                    if (lp.trail_i8[st].gemm.ntasks <= 0)
                        for (const Launch& l : lp.far[st]) add(l);
                if (lp.outer_i8.empty())
                    for (const Launch& l : lp.outer) add(l);
                for (const I8Launch& t : lp.outer_i8) {
                    add(t.gemm);
                    for (const Launch& l : t.rest) add(l);
                }
            } else {
                for (const auto& v : lp.far_tc)
                    for (const TcLaunch& t : v) add(t.gemm);
                for (const TcLaunch& t : lp.outer_tc) add(t.gemm);
            }
        }
        int64_t bad = 0;
        for (int64_t js = 0; js < ns; ++js) {
            if (P.F[js] <= kSmallMaxF) continue;
            const int32_t F = P.F[js], S = P.S[js];
            auto& c = cov[js];
            if (c.empty()) c.resize(F);
            for (int32_t col = 0; col < F; ++col) {
                // a retained front receives no update at all
                const int32_t want = P.retained[js] ? 0 : col < S ? (col / kNB) * kNB : S;
                auto& v = c[col];
                std::sort(v.begin(), v.end());
                int32_t at = 0;
                bool ok = true;
                for (const auto& iv : v) {
                    if (iv.first != at || iv.second <= iv.first) {
                        ok = false;
                        break;
                    }
                    at = iv.second;
                }
                if (!ok || at != want) ++bad;
            }
        }
        (which == 1 ? tc : fp64) += bad;
    }
}


// ---------------------------------------------------------------------------
// Stream-schedule check of the factorisation (a race detector on the host).
//
// Replays the launch order of a factorisation without hooks, all levels in turn, on
// four streams.  Per level: the small fronts by size classes on the side and
// the look-ahead stream (the first on the main one where there is no large
// front), joined at the level's end; the assembly of the large ones; per panel
// step the TRSM, the update of the next panel's columns by this panel and the
// one before and the next diagonal block on the main stream; inside a
// super-panel the update of the columns after the next two panels on the
// look-ahead stream, forked by an event after the step and joined before the
// step after the next; at the end of a super-panel the far columns' update on
// the side stream, forked by an event after the step's TRSM (as integer-digit
// update: after the split, whose slab the far launch shares) and joined before the next
// trailing update (every kSuperPanel / kNB steps) and before the K = S update; the
// write-back on a stream of its own, joined two levels later.  Vector clocks give
// the happens-before order.  Per large front it counts
//   * a panel whose columns have not received exactly the K ranges [0, k0)
//     from updates ordered before it, or that an unordered update writes;
//   * an update whose K panel columns are not final (diagonal block + TRSM
//     ordered before it);
//   * two updates on different streams that write a common element unordered;
//   * an update of the S columns not ordered before the write-back;
// and over all of the factorisation
//   * a child's update block read before its last write;
//   * a buffer written while a launch on the front that had the memory before is
//     unordered with it, or such a launch issued later;
//   * a digit slab written while a product that reads it is unordered with the
//     split, or read by a product that its own split does not precede.
// (The copy of the next panel's rows in the fronts' upper triangles is written and
// read on the main stream alone.  With hooks the small fronts and the write-back are on
// the main stream as well.)
// ---------------------------------------------------------------------------
namespace {
constexpr int kStreams = 4;          // 0 main, 1 side (far columns), 2 look-ahead, 3 write-back
struct Clock {
    int64_t t[kStreams] = {};
};
struct SchedOp {
    int stream;
    Clock vc;                        // vector clock after the op
    int32_t c0, c_end, r0, r_end;    // written block (columns, rows)
    int32_t k_lo, k_hi;              // K range applied (updates)
    int kind;                        // 0 panel, 1 update, 2 write-back
};
bool hb(const SchedOp& a, const SchedOp& b) { return a.vc.t[a.stream] <= b.vc.t[a.stream]; }

struct Replay {
    const Plan& P;
    int64_t bad = 0, reused = 0;
    Clock vc[kStreams];                                // per stream
    std::vector<Clock> touched, written;             // per front: last launch of each stream that reads or writes its buffer / writes it
    std::vector<uint8_t> gone;                       // its memory has another front's data
    std::map<int64_t, std::pair<int64_t, int32_t>> room;   // arena: first double -> (end, front)
    std::map<int32_t, std::vector<SchedOp>> ops;     // of the level's large fronts, in issue order

    explicit Replay(const Plan& p) : P(p), touched(p.nsuper), written(p.nsuper), gone(p.nsuper, 0) {}
    void wait(int dst, const Clock& ev) {
        for (int q = 0; q < kStreams; ++q) vc[dst].t[q] = std::max(vc[dst].t[q], ev.t[q]);
    }
    bool after(int stream, const Clock& last) const {
        for (int q = 0; q < kStreams; ++q)
            if (last.t[q] > vc[stream].t[q]) return false;
        return true;
    }
    void tick(int stream) { ++vc[stream].t[stream]; }
    void touch(int32_t js, int stream, bool write) {
        if (gone[js]) ++bad;
        touched[js].t[stream] = vc[stream].t[stream];
        if (write) written[js].t[stream] = vc[stream].t[stream];
    }
    // a front's first launch: its memory, and its children's update blocks
    void begin(int32_t js, int stream) {
        const int64_t lo = P.buf_off[js], hi = lo + buffer_doubles(P, js);
        if (hi > lo) {
            auto it = room.upper_bound(lo);
            if (it != room.begin() && std::prev(it)->second.first > lo) --it;
            while (it != room.end() && it->first < hi) {
                const int64_t from = it->first, to = it->second.first;
                const int32_t was = it->second.second;
                if (!gone[was]) ++reused;
                if (!after(stream, touched[was])) ++bad;
                gone[was] = 1;
                it = room.erase(it);
                if (from < lo) room[from] = {lo, was};
                if (to > hi) it = room.emplace(hi, std::make_pair(to, was)).first;
            }
            room[lo] = {hi, js};
        }
        for (int32_t k = P.child_ptr[js]; k < P.child_ptr[js + 1]; ++k) {
            const int32_t c = P.child[k];
            if (P.F[c] <= P.S[c]) continue;
            if (!after(stream, written[c])) ++bad;
            touch(c, stream, false);
        }
        touch(js, stream, true);
    }
    void issue(int stream, const Job& j, int kind) {
        SchedOp o;
        o.stream = stream;
        o.vc = vc[stream];
        o.kind = kind;
        o.k_lo = j.k_lo;
        o.k_hi = j.k_hi;
        o.c0 = o.r0 = kind == 0 ? j.k_lo : kind == 1 ? j.c0 : 0;     // a panel: columns [k_lo, k_hi), rows to F
        o.c_end = kind == 0 ? j.k_hi : j.c_end;
        o.r_end = j.r_end;
        ops[j.node].push_back(o);
        touch(j.node, stream, kind != 2);
    }
    void launch(int stream, const Launch& l, int kind) {
        tick(stream);
        for (int64_t k = 0; k < l.job_count; ++k) issue(stream, P.jobs[l.job_begin + k], kind);
    }
    void fronts();
};

// the order of the launches on each of a level's large fronts
void Replay::fronts() {
    for (auto& kv : ops) {
        const std::vector<SchedOp>& v = kv.second;
        for (size_t a = 0; a < v.size(); ++a) {
            const SchedOp& A = v[a];
            if (A.kind == 0) {
                // columns [k0, k0 + nb): K coverage [0, k0) from updates ordered before
                for (int32_t c = A.c0; c < A.c_end; ++c) {
                    std::vector<std::pair<int32_t, int32_t>> iv;
                    for (const SchedOp& U : v) {
                        if (U.kind != 1 || c < U.c0 || c >= U.c_end) continue;
                        if (!hb(U, A)) {
                            ++bad;
                            continue;
                        }
                        iv.emplace_back(U.k_lo, U.k_hi);
                    }
                    std::sort(iv.begin(), iv.end());
                    int32_t at = 0;
                    bool ok = true;
                    for (const auto& x : iv) {
                        if (x.first != at) ok = false;
                        at = x.second;
                    }
                    if (!ok || at != A.c0) ++bad;
                }
            } else if (A.kind == 1) {
                // its K panel columns are final before it
                for (const SchedOp& Q : v)
                    if (Q.kind == 0 && Q.c0 < A.k_hi && A.k_lo < Q.c_end && !hb(Q, A)) ++bad;
                // no unordered writer of a common element on another stream
                for (size_t b = a + 1; b < v.size(); ++b) {
                    const SchedOp& B = v[b];
                    if (B.kind != 1 || B.stream == A.stream) continue;
                    const bool cols = A.c0 < B.c_end && B.c0 < A.c_end;
                    const bool rows = A.r0 < B.r_end && B.r0 < A.r_end;
                    if (cols && rows && !hb(A, B) && !hb(B, A)) ++bad;
                }
            } else {
                for (const SchedOp& U : v)
                    if (U.kind == 1 && U.c0 < A.c_end && !hb(U, A)) ++bad;
            }
        }
    }
    ops.clear();
}
}  // namespace

// number of tasks of job j of launch l
static int64_t job_tasks(const Plan& P, const Launch& l, int64_t j) {
    const int64_t t0 = P.jobs[l.job_begin + j].task0;
    const int64_t t1 = (j + 1 < l.job_count) ? P.jobs[l.job_begin + j + 1].task0 : l.ntasks;
    return t1 - t0;
}

// disjoint half-open ranges inside [0, cap): the number of ranges that are not
static int64_t range_faults(std::vector<std::pair<int64_t, int64_t>> iv, int64_t cap) {
    int64_t bad = 0;
    for (const auto& r : iv)
        if (r.first < 0 || r.second > cap) ++bad;
    std::sort(iv.begin(), iv.end());
    for (size_t k = 1; k < iv.size(); ++k)
        if (iv[k].first < iv[k - 1].second) ++bad;
    return bad;
}

int64_t check_solve_plan(const Plan& P, int plant, int64_t* tasks) {
    const int64_t ns = P.nsuper;
    // the two arrays a planted mistake changes, as copies
    std::vector<int32_t> tt = P.tri_tasks;
    std::vector<int64_t> fo = P.fwd_off;
    if (plant == 1) {                      // swap blocks 0 and 1 of the first front with two blocks
        bool done = false;
        for (const LevelPlan& lp : P.levels) {
            for (int64_t t = lp.tri_begin; t < lp.tri_begin + lp.tri_count && !done; ++t) {
                if (tt[2 * t + 1] != 0) continue;
                for (int64_t u = t + 1; u < lp.tri_begin + lp.tri_count; ++u)
                    if (tt[2 * u] == tt[2 * t] && tt[2 * u + 1] == 1) {
                        std::swap(tt[2 * t + 1], tt[2 * u + 1]);
                        done = true;
                        break;
                    }
            }
            if (done) break;
        }
        if (!done) return -1;
    } else if (plant == 2) {               // one front's forward partials onto another's
        bool done = false;
        for (const LevelPlan& lp : P.levels) {
            int32_t first = -1;
            for (int32_t js : lp.elim_nodes) {
                if (P.F[js] <= P.S[js]) continue;
                if (first < 0) {
                    first = js;
                } else {
                    fo[js] = fo[first];
                    done = true;
                    break;
                }
            }
            if (done) break;
        }
        if (!done) return -1;
    } else if (plant != 0) {
        return -1;
    }
    int64_t bad = 0, nt = 0;
    // solved rows: the equations of each eliminated large front, disjoint
    {
        std::vector<std::pair<int64_t, int64_t>> iv;
        for (const LevelPlan& lp : P.levels)
            for (int32_t js : lp.elim_nodes) iv.emplace_back(P.fst[js], (int64_t)P.fst[js] + P.S[js]);
        bad += range_faults(iv, P.neq);
    }
    for (const LevelPlan& lp : P.levels) {
        // triangle tasks: each block once, after the block above it
        std::vector<int64_t> first(ns, -1);             // first block-position slot of each front
        std::vector<int64_t> pos;
        for (int32_t js : lp.elim_nodes) {
            first[js] = (int64_t)pos.size();
            pos.resize(pos.size() + (P.S[js] + kNB - 1) / kNB, -1);
        }
        if (lp.tri_begin < 0 || 2 * (lp.tri_begin + lp.tri_count) > (int64_t)tt.size()) {
            ++bad;
            continue;
        }
        for (int64_t t = lp.tri_begin; t < lp.tri_begin + lp.tri_count; ++t) {
            ++nt;
            const int32_t js = tt[2 * t], b = tt[2 * t + 1];
            if (js < 0 || js >= ns || first[js] < 0 || b < 0 || b >= (P.S[js] + kNB - 1) / kNB) {
                ++bad;
                continue;
            }
            int64_t& at = pos[first[js] + b];
            if (at >= 0) ++bad;                                          // listed twice
            at = t;
            if (b > 0 && pos[first[js] + b - 1] < 0) ++bad;              // before the block above it
        }
        for (int64_t v : pos)
            if (v < 0) ++bad;                                            // a block never listed
        // rectangles: one job per sweep and front with F > S, of the right sizes,
        // with disjoint partial-sum ranges
        std::vector<int64_t> nrect(ns, 0), nback(ns, 0), nrows(ns, 0);
        std::vector<std::pair<int64_t, int64_t>> riv, fiv;
        auto check_rect = [&](const Launch& l, std::vector<int64_t>& count, int64_t tc, bool fwd) {
            for (int64_t j = 0; j < l.job_count; ++j) {
                const Job& jb = P.jobs[l.job_begin + j];
                const int32_t js = jb.node;
                if (js < 0 || js >= ns || first[js] < 0) {
                    ++bad;
                    continue;
                }
                const int64_t f = P.F[js], s = P.S[js], tr = fwd ? fwd_rows((int)s) : kRectRows;
                const int64_t nrc = (f - s + tr - 1) / tr, ncc = (s + tc - 1) / tc;
                if (f <= s || jb.k_lo != nrc || jb.k_hi != ncc || job_tasks(P, l, j) != nrc * ncc) ++bad;
                ++count[js];
                if (fwd) fiv.emplace_back(fo[js], fo[js] + ncc * (f - s));
                else riv.emplace_back(P.rect_off[js], P.rect_off[js] + nrc * s);
            }
        };
        check_rect(lp.rect, nrect, kFwdCols, true);
        check_rect(lp.rect_back, nback, kRectCols, false);
        for (int64_t j = 0; j < lp.rect_rows.job_count; ++j) {
            const Job& jb = P.jobs[lp.rect_rows.job_begin + j];
            const int32_t js = jb.node;
            if (js < 0 || js >= ns || first[js] < 0) {
                ++bad;
                continue;
            }
            if (job_tasks(P, lp.rect_rows, j) != (int64_t)P.F[js] - P.S[js]) ++bad;
            ++nrows[js];
        }
        for (int32_t js : lp.elim_nodes) {
            const int64_t want = P.F[js] > P.S[js] ? 1 : 0;
            if (nrect[js] != want || nback[js] != want || nrows[js] != (P.S[js] > kFwdCols ? want : 0)) ++bad;
        }
        bad += range_faults(riv, P.rect_entries);
        bad += range_faults(fiv, P.fwd_entries);
    }
    if (tasks) *tasks = nt;
    return bad;
}

int64_t check_schedule(const Plan& P, bool tc, double int_min, int skip, SchedCounts* counts) {
    constexpr size_t kSteps = kSuperPanel / kNB;
    Replay R(P);
    SchedCounts n;
    Clock far_done, ahead_done[2], wb_done[2];
    bool far_open = false, ahead_open[2] = {false, false}, wb_open[2] = {false, false};
    bool far_digits = false;                             // the open far launch reads the digit slab
    auto join_far = [&]() {
        if (far_open && !(skip & kSkipFar)) R.wait(0, far_done);
        far_open = false;
    };
    auto join_ahead = [&](size_t st) {
        if (ahead_open[st & 1] && !(skip & kSkipAhead)) R.wait(0, ahead_done[st & 1]);
        ahead_open[st & 1] = false;
    };
    // the digit slab: its split, that split's place on the main stream, its readers
    const I8Launch* slab_of = nullptr;
    int64_t slab_at = 0;
    Clock slab_read;
    auto split = [&](const I8Launch& t) {
        R.tick(0);
        for (int64_t k = 0; k < t.split.job_count; ++k) R.touch(P.jobs[t.split.job_begin + k].node, 0, false);
        if (!R.after(0, slab_read)) ++R.bad;
        slab_of = &t;
        slab_at = R.vc[0].t[0];
    };
    auto product = [&](int stream, const I8Launch& t, const Launch& l) {
        R.launch(stream, l, 1);
        if (slab_of != &t || slab_at > R.vc[stream].t[0]) ++R.bad;
        slab_read.t[stream] = R.vc[stream].t[stream];
    };
    for (size_t L = 0; L < P.levels.size(); ++L) {
        const LevelPlan& lp = P.levels[L];
        if (wb_open[L & 1] && !(skip & kSkipWriteback)) R.wait(0, wb_done[L & 1]);
        wb_open[L & 1] = false;
        // small fronts
        const int small[2] = {lp.large_nodes.empty() ? 0 : 1, lp.small_classes.size() > 1 ? 2 : 0};
        const bool beside = !lp.small_classes.empty() && (small[0] || small[1]);
        n.small_beside += beside;
        if (!lp.small_classes.empty())
            for (int t : small) R.wait(t, R.vc[0]);
        for (size_t c = 0; c < lp.small_classes.size(); ++c) {
            R.tick(small[c & 1]);
            for (int32_t k = 0; k < lp.small_classes[c].count; ++k)
                R.begin(lp.small_nodes[lp.small_classes[c].begin + k], small[c & 1]);
        }
        auto join_small = [&]() {
            if (beside && !(skip & kSkipSmall))
                for (int t : small) R.wait(0, R.vc[t]);
        };
        if (lp.large_nodes.empty()) {
            join_small();
            continue;
        }
        // large fronts
        R.tick(0);
        for (int32_t js : lp.large_nodes) R.begin(js, 0);
        for (size_t st = 0; st < lp.panel.size(); ++st) {
            // a super-panel's first diagonal block, then the TRSM, the next panel's columns
            // and its diagonal block
            const Launch& pl = lp.panel[st];
            const bool chain = (st + 1) % kSteps != 0;
            if (st % kSteps == 0) R.launch(0, pl, 0);
            join_ahead(st);
            R.launch(0, pl, 0);
            if (chain)
                for (int64_t k = 0; k < pl.job_count; ++k) {
                    const Job c = chain_update(P, P.jobs[pl.job_begin + k]);
                    if (c.c0 >= c.c_end) continue;
                    R.tick(0);
                    R.issue(0, c, 1);
                    Job d = c;
                    d.k_lo = c.c0;
                    d.k_hi = c.c_end;
                    R.tick(0);
                    R.issue(0, d, 0);
                }
            const bool has_far = !lp.far[st].empty() || !lp.far_tc[st].empty();
            const I8Launch& t = lp.trail_i8[st];
            const bool digits = !tc && t.gemm.ntasks > 0 && t.flops >= int_min;
            if (has_far && !digits) R.wait(1, R.vc[0]);  // fork after the step's TRSM
            n.slab_shared += digits && far_open && far_digits;
            if (digits && (skip & kSkipSlab)) split(t);
            if (!chain) join_far();
            const Clock fork = R.vc[0];
            if (digits) {
                if (!(skip & kSkipSlab)) split(t);
                if (has_far) R.wait(1, R.vc[0]);
                product(0, t, t.gemm);
                for (const Launch& ul : t.rest) R.launch(0, ul, 1);
            } else {
                for (const Launch& ul : lp.update[st]) R.launch(0, ul, 1);
            }
            if (!lp.ahead[st].empty()) {
                R.wait(2, fork);
                for (const Launch& al : lp.ahead[st]) R.launch(2, al, 1);
                ahead_done[st & 1] = R.vc[2];
                ahead_open[st & 1] = true;
            }
            if (has_far) {
                far_digits = digits && t.far.ntasks > 0;
                if (digits) {
                    if (far_digits) product(1, t, t.far);
                    for (const Launch& fl : t.far_rest) R.launch(1, fl, 1);
                } else if (tc) {
                    for (const TcLaunch& f : lp.far_tc[st]) R.launch(1, f.gemm, 1);
                } else {
                    for (const Launch& fl : lp.far[st]) R.launch(1, fl, 1);
                }
                far_done = R.vc[1];
                far_open = true;
            }
        }
        join_ahead(0);
        join_ahead(1);
        join_far();
        R.wait(3, R.vc[0]);
        R.tick(3);
        for (int32_t js : lp.large_nodes) {
            if (P.retained[js]) R.touch(js, 3, false);
            else R.issue(3, Job{js, 0, P.S[js], P.F[js], 0, 0, 0}, 2);
        }
        wb_done[L & 1] = R.vc[3];
        wb_open[L & 1] = true;
        if (tc) {
            for (const TcLaunch& t : lp.outer_tc) R.launch(0, t.gemm, 1);
        } else if (!lp.outer_i8.empty() && lp.outer_i8[0].flops >= int_min) {
            for (const I8Launch& t : lp.outer_i8) {
                if (t.gemm.ntasks > 0) {
                    split(t);
                    product(0, t, t.gemm);
                }
                for (const Launch& ol : t.rest) R.launch(0, ol, 1);
            }
        } else {
            for (const Launch& ol : lp.outer) R.launch(0, ol, 1);
        }
        join_small();
        R.fronts();
    }
    n.reused = R.reused;
    if (counts) *counts = n;
    return R.bad;
}

uint64_t sm_hash_host(const double* a, int64_t n, int threads) {
    const uint64_t* w = reinterpret_cast<const uint64_t*>(a);
    auto part = [w](int64_t i0, int64_t i1) {
        uint64_t acc = 0;
        for (int64_t i = i0; i < i1; ++i) acc += sm_mix(w[i], (uint64_t)i);
        return acc;
    };
    const int64_t per = int64_t(1) << 22;             // below 32 MB one thread is enough
    int nt = (int)std::min<int64_t>(std::max(threads, 1), (n + per - 1) / per);
    if (nt <= 1) return part(0, n);
    std::vector<uint64_t> sums(nt, 0);
    std::vector<std::thread> pool;
    for (int t = 0; t < nt; ++t)
        pool.emplace_back([&, t]() { sums[t] = part(n * t / nt, n * (t + 1) / nt); });
    for (auto& th : pool) th.join();
    uint64_t h = 0;
    for (uint64_t v : sums) h += v;
    return h;
}

}  // namespace sprb
