"""The flat work lists of the FP64 evaluation pass (csrc/plan.cpp, compiled here
without a GPU): over tree and degree edges, every list entry's sources are in its
target set's stages exactly once (single-tree lists: for exactly the targets that
list them), stages and units are well formed, partial sums do not overlap, and the
leaves' ends name every target slot above them.  Single-tree plans hold none of the
batched form's work lists, only their count.
"""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sal-fort_b200", "csrc")

PROGRAM = r"""
#include "sal_internal.hpp"
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <random>
using namespace sal;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)
int main(int, char **v) {
    const int stt = atoi(v[1]), n = atoi(v[2]), thresh = atoi(v[3]), d = atoi(v[4]), P = (d + 1) * (d + 1);
    std::mt19937 rng(n);
    std::normal_distribution<double> g;
    std::vector<double> x(n), y(n), z(n);
    for (int i = 0; i < n; ++i) {
        const double a = g(rng), b = g(rng), c = g(rng), r = std::sqrt(a * a + b * b + c * c);
        x[i] = a / r; y[i] = b / r; z[i] = c / r;
    }
    Tree *t = tree_build(x.data(), y.data(), z.data(), n, thresh);
    std::vector<int32_t> L, pc, pp;
    if (stt) single_tree_traversal(*t, 0.7, thresh, x.data(), y.data(), z.data(), n, &pc, &pp);
    else L = dual_tree_traversal(*t, 0.7, thresh);
    Plan pl;
    std::string err;
    CHECK(plan_build(*t, x.data(), y.data(), z.data(), d, stt, L.data(), (int64_t)L.size() / 3, pc.data(),
                     (int64_t)pc.size() / 2, pp.data(), (int64_t)pp.size() / 2, &pl, &err));
    std::vector<int32_t> slot(t->p.size(), -1), tslot(t->p.size(), -1), pos(n);
    for (size_t s = 0; s < pl.src_slot_panel.size(); ++s) slot[pl.src_slot_panel[s]] = (int32_t)s;
    for (size_t s = 0; s < pl.tgt_slot_panel.size(); ++s) tslot[pl.tgt_slot_panel[s]] = (int32_t)s;
    for (int p = 0; p < n; ++p) pos[t->order[p]] = p;
    // want[target: pool position, or n + slot][first source row]: how often
    std::map<std::pair<int, int>, int> want, have;
    auto first = [&](int k, int kind) { return kind ? n + slot[k] * P : (int)t->p[k].begin; };
    for (size_t i = 0; i + 2 < L.size(); i += 3) {
        const int kt = L[i] - 1, ks = L[i + 1] - 1, ty = L[i + 2], f = first(ks, ty & 1);
        if (!t->p[kt].count() || !t->p[ks].count()) continue;
        for (int r = 0; r < (ty & 1 ? P : (int)t->p[ks].count()); ++r) {
            if (ty >= 2) ++want[{n + tslot[kt], f + r}];
            else for (int64_t p = t->p[kt].begin; p < t->p[kt].end; ++p) ++want[{(int)p, f + r}];
        }
    }
    std::map<std::pair<int, int>, bool> listed;   // (leaf's first row, source): one item per kMaxStage of them
    int64_t pieces = 0;
    std::vector<int> leaf_of(n);
    for (const Panel &q : t->p)
        if (q.is_leaf) for (int64_t p = q.begin; p < q.end; ++p) leaf_of[p] = (int)q.begin;
    for (int kind = 0; kind < 2; ++kind) {
        const auto &l = kind ? pc : pp;
        for (size_t i = 0; i + 1 < l.size(); i += 2) {
            const int p = pos[l[i] - 1], ks = l[i + 1] - 1, f = first(ks, kind), c = kind ? P : (int)t->p[ks].count();
            for (int r = 0; r < c; ++r) want[{p, f + r}] = 1;
            bool &seen = listed[{leaf_of[p], ks * 2 + kind}];
            if (!seen) pieces += (c + kMaxStage - 1) / kMaxStage;
            seen = true;
        }
    }
    if (stt) CHECK(pl.leaf_items.empty() && pl.leaf_groups.empty() && pl.list_items == pieces);
    else CHECK(pl.list_items == (int64_t)pl.leaf_items.size());
    std::vector<int> row(pl.leaf_part_rows, 0), stage(pl.eval_stages.size(), 0), item(pl.eval_items.size(), 0);
    std::map<int, int> straight, punit;
    for (size_t k = 0; k < pl.eval_units.size(); ++k) {
        const EvalUnit &u = pl.eval_units[k];
        CHECK((u.proxy != 0) == ((int)k < pl.n_proxy_eval));
        CHECK(u.sb <= u.sm && u.sm <= u.se && u.nt >= 1 && u.nt <= 256);
        if (u.proxy) {
            CHECK(pl.eval_proxy_unit_beg[u.tgt] <= u.out && u.out < pl.eval_proxy_unit_beg[u.tgt + 1]);
            CHECK(++punit[u.out] == 1);
        } else if (u.out < 0) {
            CHECK(++straight[u.tgt] == 1);
        } else {
            for (int i = 0; i < u.nt; ++i) ++row[u.out + i];
        }
        for (int s = u.sb; s < u.se; ++s) {
            const EvalStage &S = pl.eval_stages[s];
            ++stage[s];
            CHECK(S.cnt >= 1 && S.cnt <= kMaxStage && S.ie - S.ib >= 1 && S.ie - S.ib <= kStageItems);
            int at = 0;
            for (int i = S.ib; i < S.ie; ++i) {
                const EvalItem &it = pl.eval_items[i];
                ++item[i];
                CHECK(it.dst == at && it.cnt >= 1 && (it.mask >= 0) == !!(S.flags & kEvalMasked));
                at += it.cnt;
                if (stt) CHECK((it.off >= n) == (s >= u.sm));
                for (int j = 0; j < u.nt; ++j) {
                    if (it.mask >= 0 && !((pl.masks[it.mask + j / 32] >> (j % 32)) & 1u)) continue;
                    if (u.proxy && j) break;
                    for (int r = 0; r < it.cnt; ++r) ++have[{u.proxy ? n + u.tgt : u.tgt + j, it.off + r}];
                }
            }
            CHECK(at == S.cnt);
        }
    }
    CHECK(want == have);
    for (int r : row) CHECK(r == 1);
    for (int s : stage) CHECK(s == 1);
    for (int i : item) CHECK(i == 1);
    int64_t down = 0, part = 0;
    for (const LeafFin &f : pl.leaf_fin) {
        CHECK(!straight.count(f.tgt) && f.db == down && f.part == part);
        std::vector<int32_t> above;
        for (size_t s = 0; s < pl.tgt_slot_panel.size(); ++s) {
            const Panel &q = t->p[pl.tgt_slot_panel[s]];
            if (q.begin <= f.tgt && f.tgt < q.end) above.push_back((int32_t)s);
        }
        CHECK(std::vector<int32_t>(pl.down_slots.begin() + f.db, pl.down_slots.begin() + f.de) == above);
        down = f.de;
        part += (int64_t)f.parts * f.nt;
    }
    CHECK(down == (int64_t)pl.down_slots.size() && part == pl.leaf_part_rows);
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan_eval.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-std=c++17", "-fopenmp", "-ffp-contract=off", "-I/usr/local/cuda/include", "-I", CSRC,
                    str(d / "plan_eval.cpp"), os.path.join(CSRC, "plan.cpp"), os.path.join(CSRC, "tree.cpp"),
                    "-o", str(d / "plan_eval")], check=True)
    return str(d / "plan_eval")


@pytest.mark.parametrize("stt,n,thresh,degree", [(0, 6, 2, 1), (0, 240, 257, 8), (0, 1500, 7, 2), (0, 3000, 100, 8),
                                                 (0, 2500, 257, 14), (1, 240, 257, 8), (1, 1500, 7, 2), (1, 2500, 60, 8),
                                                 (2, 2500, 257, 14)])
def test_eval_lists(program, stt, n, thresh, degree):
    r = subprocess.run([program, str(stt), str(n), str(thresh), str(degree)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
