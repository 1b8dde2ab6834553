"""The host arithmetic of the attention kernels (tessera_b200/csrc/attention_plan.h), compiled by the host compiler and
compared with the rules stated here."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    """plan(expression, ...) -> the values the expressions have in C++."""
    where = tmp_path_factory.mktemp("plan")

    def values(*expressions):
        source = '#include <cstdio>\n#include "attention_plan.h"\nusing namespace tsr;\nint main() {\n'
        source += "".join('  std::printf("%%lld\\n", static_cast<long long>(%s));\n' % e for e in expressions) + "}\n"
        (where / "p.cpp").write_text(source)
        subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-fsanitize=undefined", "-fno-sanitize-recover", "-I",
                        os.path.join(ROOT, "tessera_b200", "csrc"), str(where / "p.cpp"), "-o", str(where / "p")], check=True)
        out = subprocess.run([str(where / "p")], check=True, capture_output=True, text=True).stdout
        return [int(x) for x in out.split()]
    return values


def walked(m, n, q_base, window, group):
    """Keys of the row tile that walks over most of them, row by row."""
    pairs, most = [(i, g) for i in range(m) for g in range(group)], 0
    for t in range(0, len(pairs), 128):
        rows = {i for i, _ in pairs[t:t + 128]}
        last = max(min(q_base + i, n - 1) for i in rows)
        start = min(min(max(0, q_base + i + 1 - window), min(q_base + i, n - 1)) if window else 0 for i in rows)
        most = max(most, last - start + 1)
    return most


@pytest.mark.parametrize("group", [1, 2, 5, 6, 7, 8])
def test_span_covers_every_row_tile(plan, group):
    cases = [(m, n, b, w) for m in (1, 4, 60, 300) for n in (70, 700) for b in (0, 33, n - 1, n + 5)
             for w in (0, 1, 50, 650, 2**31 - 1)]
    spans = plan(*("tile_span(%d, %d, %dull, %d, true, %d)" % (*c, group) for c in cases))
    for (m, n, b, w), span in zip(cases, spans):
        assert walked(m, n, b, w, group) <= span <= n, (m, n, b, w)


def test_widest_window_and_no_mask(plan):
    """A window beyond every position is no window, up to the largest the entry points take."""
    wide = ["tile_span(512, 4096, 3584, %d, true, %d)" % (w, g) for w in (2**31 - 1, 2**31 - 18, 4096) for g in (1, 6, 8)]
    assert plan(*wide, "tile_span(8, 500, 0, 3, false, 2)") == [4096] * len(wide) + [500]


def cluster_plan(span, clusters, resident):
    """(CTAs per cluster, one wave) by the rule."""
    most = 1
    while most < 16 and most * 16 < span:
        most *= 2
    sizes = [c for c in (16, 8, 4, 2, 1) if c <= most and clusters <= resident[c]]
    return (sizes[0], 1) if sizes else (min(most, 8), 0)


# clusters of 1, 2, 4, 8, 16 CTAs that run at a time: a whole B200, one that takes no clusters of sixteen, a small partition
DEVICES = [{1: 148, 2: 74, 4: 36, 8: 14, 16: 7}, {1: 148, 2: 74, 4: 36, 8: 14, 16: 0}, {1: 14, 2: 7, 4: 3, 8: 1, 16: 0}]


@pytest.mark.parametrize("resident", DEVICES)
def test_clusters_of_few_rows(plan, resident):
    """A size the device does not take is never chosen, nor a reason to refuse a call that smaller ones serve; one that is
    not needed is not asked for."""
    cases = [(s, c) for s in (1, 16, 17, 100, 129, 4096, 2**31 - 1) for c in (1, 4, 7, 8, 14, 15, 36, 37, 100, 148, 149, 60000)]
    lookup = "[&](int c) { asked = c > asked ? c : asked; return c == 1 ? %d : c == 2 ? %d : c == 4 ? %d : c == 8 ? %d : %d; }" % tuple(
        resident[c] for c in (1, 2, 4, 8, 16))
    got = plan(*("[] { int asked = 0; bool w; const int c = few_ctas(%d, %d, %s, &w); return c + 100 * w + 1000 * asked; }()" % (s, c, lookup)
                 for s, c in cases))
    for (span, clusters), v in zip(cases, got):
        want, wave = cluster_plan(span, clusters, resident)
        assert v % 100 == want and v // 100 % 10 == wave, (span, clusters)
        assert v // 1000 <= max(1, 2 * span / 16)
        assert resident[want] > 0


def test_kernel_for_a_batch(plan):
    """All clusters at a time and 512 keys of 256 elements a CTA (256 with one or two CTAs a cluster); fp16 row tiles."""
    wins = [("4096, 8, true, 256", 1), ("4097, 8, true, 256", 0), ("8192, 8, true, 128", 1), ("512, 2, true, 256", 1), ("513, 2, true, 256", 0),
            ("16, 1, true, 256", 1), ("16, 1, false, 256", 0), ("2147483647, 16, true, 256", 0)]
    assert plan(*("few_rows_win(%s)" % a for a, _ in wins)) == [v for _, v in wins]
    assert plan("tile_least(false, 4)", "tile_least(true, 4)", "tile_least(true, 16)") == [12000000, 45000000, 22000000]
