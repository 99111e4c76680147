"""The end of a TMA staging ring whose block gives up (csrc/fr_ring.h), on the CPU against a model
of the slots' barriers: whatever was issued, whatever has landed and wherever the waits stopped,
drain_fills returns only when every issued copy has landed, so none writes into
shared memory that its block no longer owns.  The staged kernels are read for the other half: each ends
its ring by the number of fills it issued, the gradient's filling warp on every path."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fastreg_gb300" / "csrc"

MODEL = r"""
#include "fr_ring.h"
#include <cstdio>
#include <vector>

// Barriers whose phase k of slot s completes when the slot's k-th fill lands; a wait for a parity passes when
// the phase under way has the other one (mbarrier.try_wait.parity).
template <int S>
int check() {
    typedef frg::SliceRing<S> Ring;
    for (unsigned issued = 0; issued <= 5u * S + 1; ++issued) {
        const unsigned flying = issued < (unsigned)S ? issued : (unsigned)S;  // only the last S can be in flight
        for (unsigned mask = 0; mask < (1u << flying); ++mask) {             // bit j: fill issued - flying + j has landed
            std::vector<char> landed(issued, 1);
            std::vector<unsigned> done(S, 0);
            for (unsigned j = 0; j < flying; ++j) landed[issued - flying + j] = (mask >> j) & 1;
            for (unsigned n = 0; n < issued; ++n) done[Ring::slot(n)] += landed[n];
            int ran_out = 0;
            frg::drain_fills<S>(issued, [&](int k, unsigned parity) {
                if ((done[k] & 1u) != parity) return;
                for (unsigned n = k; n < issued; n += S)
                    if (!landed[n]) {  // the wait lasts until this copy lands
                        landed[n] = 1;
                        ++done[k];
                        return;
                    }
                ++ran_out;  // a wait for a fill that was never issued
            });
            for (unsigned n = 0; n < issued; ++n)
                if (!landed[n]) return std::printf("S=%d issued=%u mask=%x: fill %u in flight\n", S, issued, mask, n), 1;
            if (ran_out) return std::printf("S=%d issued=%u mask=%x: %d waits ran out\n", S, issued, mask, ran_out), 1;
        }
    }
    return 0;
}
int main() { return check<3>() | check<4>() | check<6>(); }
"""


def test_every_issued_copy_lands_before_a_block_ends(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    (tmp_path / "ring.cpp").write_text(MODEL)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(CSRC), str(tmp_path / "ring.cpp"), "-o", str(tmp_path / "ring")],
                   check=True)
    r = subprocess.run([str(tmp_path / "ring")], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("name,kernel,drain", [("fr_ref.cu", "ref_laplacian_tma_kernel", "drain_fills<kTLS>(issued,"),
                                               ("fr_ref.cu", "ref_pass_a_tma_kernel", "drain_fills<kPVS>(issued,"),
                                               ("fr_sob.cu", "sob_grad_kernel", "drain_fills<kGS>(n,")])
def test_staged_kernels_end_their_ring_by_what_they_issued(name, kernel, drain):
    text = (CSRC / name).read_text()
    body = text[text.index(f" {kernel}("):]
    body = body[:re.search(r"^}$", body, re.M).end()]
    assert body.count("drain_fills<") == 1 and drain in body
    counter = drain[drain.index("(") + 1:-1]
    assert body.count(f"++{counter}") == 1  # counted where a fill is issued, nowhere else
    if kernel == "sob_grad_kernel":  # its warps may leave while the filling thread has seen no failure
        line = body[:body.index(drain)].rstrip().splitlines()
        code = [l for l in line if not l.lstrip().startswith("//")]
        assert code[-1].strip() == "}", "the filling thread drains on every path"
