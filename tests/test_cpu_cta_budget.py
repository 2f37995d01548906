"""cpdlp_submit's max_ctas caps the CTAs that a job runs at a time, over all the
launches that run side by side (csrc/cta_budget.h, built here by itself)."""
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "coolpdlp.jl_gb300", "csrc")
MAIN = r"""
#include <cstdio>
#include "cta_budget.h"
int main() {
    long cap; int n;
    while (std::scanf("%ld %d", &cap, &n) == 2) {
        std::vector<cpdlp::CtaShare> v;
        for (int k = 0; k < n; k++) {
            cpdlp::CtaShare s{1, 0, 0.0};
            long most;
            if (std::scanf("%d %ld %lf", &s.cs, &most, &s.work) != 3) return 1;
            s.most = most;
            v.push_back(s);
        }
        std::printf("%d", (int)cpdlp::share_ctas(v, cap));
        for (auto& s : v) std::printf(" %ld", (long)s.groups);
        std::printf("\n");
    }
}
"""


@pytest.fixture(scope="module")
def share(tmp_path_factory):
    d = tmp_path_factory.mktemp("budget")
    (d / "main.cpp").write_text(MAIN)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")])

    def run(cases):
        text = "\n".join(f"{cap} {len(v)} " + " ".join(f"{c} {m} {w}" for c, m, w in v) for cap, v in cases)
        out = subprocess.run([str(d / "main")], input=text, text=True, capture_output=True, check=True)
        rows = [[int(q) for q in line.split()] for line in out.stdout.splitlines()]
        return [(bool(r[0]), r[1:]) for r in rows]

    return run


def _mixes():
    """Launch sets of a mixed job: tile CTAs, tile clusters, resident classes."""
    rng = np.random.RandomState(4)
    for _ in range(300):
        v = [(1, int(rng.choice([0, 3, 200])), float(rng.rand() * 500)),
             (8, int(rng.choice([0, 1, 19])), float(rng.rand() * 500))]
        for cs in (8, 8, 8, 4, 4, 4, 2, 2, 1, 1, 1)[:rng.randint(0, 12)]:
            v.append((cs, int(rng.randint(1, 120)), float(rng.rand() * 1000)))
        yield int(rng.choice([1, 4, 7, 16, 40, 152, 100000])), v


def test_one_budget_for_all_launches(share):
    cases = list(_mixes())
    for (cap, v), (serial, groups) in zip(cases, share(cases)):
        held = [g * c for g, (c, _, _) in zip(groups, v)]
        for g, (_, most, _) in zip(groups, v):
            assert (g >= 1) == (most > 0) and g <= most
        if serial:  # one after another: each within the cap, or one cluster
            assert sum(c for c, m, _ in v if m > 0) > cap
            assert all(h <= cap or g == 1 for h, g in zip(held, groups))
        else:
            assert sum(held) <= cap
            # nothing that would still fit is left unused
            assert not any(g < m and c <= cap - sum(held) for g, (c, m, _) in zip(groups, v))


def test_no_cap_gives_every_launch_all_its_groups(share):
    v = [(1, 608, 3.0), (8, 19, 5.0), (4, 31, 1.0)]
    assert share([(0, v), (10**6, v)]) == [(False, [608, 19, 31])] * 2


def test_the_longest_work_gets_the_most(share):
    v = [(1, 500, 100.0), (8, 500, 700.0), (1, 500, 200.0)]
    (serial, groups), = share([(152, v)])
    assert not serial
    for g, (cs, _, work) in zip(groups, v):  # in proportion, to within a cluster
        assert abs(g * cs - 152 * work / 1000.0) <= 8
