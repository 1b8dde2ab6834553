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
