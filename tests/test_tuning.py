"""CPU test of the chunks that the autotuner tries (tuning.hpp): each of them makes other launches
than the default and than the others, in the accurate mode and under the bin_slop rule, and there
is something to try wherever an expansion runs."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <set>
#include "tuning.hpp"
using namespace tc;
int main()
{
    for (long long n : {300LL, 5000LL, 100003LL, 262144LL, 1000000LL, 10000000LL, 300000000LL})
        for (long long ntop : {1LL, 8LL, 64LL, 1024LL, 40000LL}) {
            const long long ngen = ntop * (ntop + 1) / 2;
            const double per = (double)n / ntop * ((double)n / ntop);
            for (int walk = 0; walk < 2; ++walk) {
                const std::vector<long long> c = tune_chunks(walk, n, ngen, per);
                auto launch = [&](long long ch) { return walk ? walk_start(ch, n, ngen, per) : ch ? ch : expand_chunk(n); };
                std::set<long long> seen = {launch(0)};
                bool ok = true;
                for (long long ch : c)
                    ok = ok && seen.insert(launch(ch)).second && ch >= 65536 && ch <= (1 << 26) && (ch & (ch - 1)) == 0;
                if (walk ? launch(0) > 0 : launch(0) > (1 << 21)) ok = ok && !c.empty();
                else ok = ok && c.empty();
                std::printf("%d %lld %lld %d %zu\n", (int)ok, n, ntop, walk, c.size());
            }
        }
}
"""


def test_every_candidate_is_another_launch(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "treecorr_gb300", "csrc"),
                    str(tmp_path / "t.cpp"), "-o", exe], check=True)
    lines = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    assert len(lines) == 70
    assert [l for l in lines if not l.startswith("1 ")] == []
    # The benchmark catalog: 10M points under 1024 top-level cells.
    assert "1 10000000 1024 1 2" in lines
