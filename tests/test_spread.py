"""How small launches lay their rays out (spread.h), compiled for the host:
for every count and number of warps, 0 warps included, the rule is defined and
the lanes or quads it names hold all rays."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aviatorengine2_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "spread.h"
int main() {
    const uint32_t most = 0xffffffffu;
    const uint32_t warps[] = {0, 1, 2, 3, 31, 32, 4735, 4736, 4737, 1u << 20, most};
    const uint32_t counts[] = {0, 1, 2, 31, 32, 33, 2368, 2369, 18944, 18945, 37888, 37889, 300001, 1u << 30, most};
    int bad = 0;
    for (uint32_t w : warps)
        for (uint32_t n : counts) {
            const uint32_t lanes = ae::spread_lanes(n, w), quads = ae::spread_quads(n, w);
            const uint64_t half = w > 1 ? (uint64_t(w) + 1) / 2 : 1;
            if (lanes < 1 || (lanes > 16 && lanes != 32) || quads > 8) bad++;
            if (lanes <= 16 && lanes * half < n) bad++;
            if (quads && quads * half < n) bad++;
            if (!quads && 8 * half >= n) bad++;
        }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_spread_rules(tmp_path):
    src, exe = tmp_path / "spread.cpp", tmp_path / "spread"
    src.write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, str(src), "-o", str(exe)])
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (out.returncode, out.stdout.strip()) == (0, "0")


def test_launchers_keep_no_plain_statics():
    """Contexts may be used by one thread each: a launcher's function statics
    are constants (initialised once, by the language), not variables that two
    threads fill."""
    import re
    found = []
    for name in sorted(os.listdir(CSRC)):
        for line in open(os.path.join(CSRC, name)):
            if re.match(r"\s+static (?!const|constexpr|thread_local|float centre|__device__)[\w:<>*]+ \w+( =|;|,|\{)", line):
                found.append((name, line.strip()))
    assert not found
