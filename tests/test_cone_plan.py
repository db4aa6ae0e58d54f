"""How the projection's boxes are laid out over blocks (csrc/cone_plan.cuh), on the CPU: the form and the words of a row
for boxes at the edges of each form, and what every plan keeps to, over random boxes."""
import random
import subprocess

import pytest

from atjup_b200 import build

SRC = r"""
#include <cstdio>
#include "cone_plan.cuh"
using namespace atjup;
// boxes from stdin, one plan a line: clusters C levels NJ NK ring n_tab ...
int main() {
    int sms, n;
    while (scanf("%d %d", &sms, &n) == 2) {
        std::vector<ConeBox> b(n);
        for (auto& x : b) if (scanf("%d %d %d %d", &x.NJ, &x.NK, &x.ring, &x.n_tab) != 4) return 1;
        const ConePlan p = cone_plan(b, [&](const ConePlan& q) { return n * q.C <= sms; });
        printf("%d %d %d %d %zu", p.C, p.row, p.smem, p.threads, p.bytes);
        for (const auto& x : b) printf(" %d", cone_words(x, p.row));
        printf("\n");
    }
}
"""
CAP, DEFAULT_SMS = 227 * 1024, 148


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "p.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-x", "c++", "-I", str(build.CSRC), "-o", str(d / "p"), str(d / "p.cpp")], check=True)

    def run(cases):
        text = "\n".join(f"{sms} {len(b)} " + " ".join(f"{x[0]} {x[1]} {x[2]} {x[3]}" for x in b) for sms, b in cases)
        out = subprocess.run([str(d / "p")], input=text, check=True, capture_output=True, text=True).stdout
        rows = [list(map(int, l.split())) for l in out.splitlines()]
        assert len(rows) == len(cases)
        return [dict(C=r[0], row=r[1], smem=r[2], threads=r[3], bytes=r[4], words=r[5:]) for r in rows]
    return run


def box(NJ, NK, n_tab=1000):
    ring = 1
    while ring < (NJ + NK - 2) // 2 + 12:
        ring *= 2
    return NJ, NK, ring, n_tab


@pytest.mark.parametrize("NJ, NK, row, words", [
    (35, 47, True, 64), (112, 125, True, 64), (8, 30, True, 64),     # bands of 2 to 28 rows, at most 64 words
    (117, 31, False, 17), (117, 60, False, 31), (117, 61, False, 32),  # more rows: one chunk of 32 words up to 61
    (117, 62, False, 32), (117, 63, False, 33),                        # meridians, two from 63
    (35, 127, False, 65), (7, 31, False, 17), (3, 31, False, 17)],     # wider rows, bands of one row
    ids=lambda v: str(v))
def test_words_of_a_row(plans, NJ, NK, row, words):
    p, = plans([(DEFAULT_SMS, [box(NJ, NK)] * 4)])
    assert p["smem"] and p["row"] == row and p["words"] == [words] * 4


def test_every_plan_keeps_its_bounds(plans):
    rng = random.Random(5)
    cases = []
    for _ in range(3000):
        n = rng.randint(1, 60)
        J, K = int(2 ** rng.uniform(0, 9)), int(2 ** rng.uniform(0, 9))
        b = [box(max(1, J - rng.randint(0, 3)), max(1, K - rng.randint(0, 3)), 2 * rng.randint(0, 4 * (J + K))) for _ in range(n)]
        cases.append((rng.choice([148, 132, 40]), b))
    seen = set()
    for (sms, b), p in zip(cases, plans(cases)):
        seen.add((p["row"], p["smem"]))
        assert 0 < p["bytes"] <= CAP and 1 <= p["C"] <= 4 and p["C"] <= min(x[0] for x in b)
        assert p["C"] == 1 or len(b) * p["C"] <= sms
        for x, words in zip(b, p["words"]):
            assert words == (64 if p["row"] else (x[1] + 3) // 2)
            assert words >= (x[1] + 3) // 2
            if p["row"]:
                assert x[0] // p["C"] >= 2 and -(-x[0] // p["C"]) <= 28 and p["threads"] >= 32 * -(-x[0] // p["C"])
    assert seen == {(1, 1), (0, 1), (0, 0)}


def test_larger_constants_keep_a_box_in_shared_memory(plans):
    """A box whose bands fit 200 KB with two doubles a special cell and six a row, up to 300 wall cells and 4000 near
    ones, runs in clusters whatever the constants take now."""
    rng = random.Random(7)
    cases, sizes = [], []
    while len(cases) < 300:
        J, K = rng.randint(40, 400), rng.randint(40, 400)
        wall, near = rng.randint(0, 300), rng.randint(0, 4000)
        rows, words, ring = -(-J // 4), (K + 3) // 2, 1
        while ring < (J + K - 2) // 2 + 2:
            ring *= 2
        small = 8 * (2 * (rows + 2) * words + 6 * J + 2 * (wall + near)) + 8 * rows * words + 16 * ring
        if 150 * 1024 < small <= 200 * 1024:
            cases.append((DEFAULT_SMS, [box(J, K, 8 * wall + 2 * near)]))
            sizes.append(small)
    assert max(sizes) > 195 * 1024
    for p in plans(cases):
        assert p["smem"] and p["C"] == 4
