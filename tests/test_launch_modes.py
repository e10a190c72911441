"""Which kernels carry the programmatic attribute and which may read ahead of their wait, in every mode of csrc/launch_mode.h (no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r'''
#include "launch_mode.h"
namespace flexllm {
thread_local LaunchMode g_pdl = kWhole;
static bool g_on = true;
bool programmatic_launches() { return g_on; }
}
using namespace flexllm;
static bool next() { const bool p = programmatic_next(); launched(); return p; }
int main() {
    if (next() || may_read_ahead() || in_chain()) return 1;
    {
        const SetUpEarly early;                                     // set up early: overlapped, but nothing is read ahead
        if (!next() || may_read_ahead() || in_chain()) return 2;
        {
            const ReadsAhead weights;                               // a kernel that reads ahead all the same is launched whole
            if (next() || may_read_ahead()) return 3;
            const SetUpEarly again;
            if (!next() || may_read_ahead()) return 4;
        }
        if (!next() || may_read_ahead()) return 5;
    }
    if (g_pdl != kWhole) return 6;
    g_pdl = kChainStart;
    if (!in_chain() || may_read_ahead() || next()) return 7;        // the first kernel of a chain
    {
        const SetUpEarly early;                                     // inside a chain neither scope changes anything
        const ReadsAhead weights;
        if (!in_chain() || !may_read_ahead() || !next()) return 8;
    }
    if (g_pdl != kChain) return 9;
    g_pdl = kWhole;
    g_on = false;
    const SetUpEarly off;
    return next() ? 10 : 0;
}
'''


def test_launch_modes(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "flexllm_b200", "csrc"), str(tmp_path / "t.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe]).returncode == 0
