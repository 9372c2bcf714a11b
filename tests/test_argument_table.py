"""What an emulated group remembers of its argument tables (csrc/gpu/arg_table.hpp), built as a host program."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include <stdexcept>
#include "gpu/arg_table.hpp"
int main() {
    cclx::gpu::arg_table t;
    const int a[2] = { 1, 2 }, b[2] = { 3, 4 };
    int copies = 0, other = 0;
    auto copy = [&] { copies++; };
    auto fail = [] { throw std::runtime_error("copy"); };
    auto fails = [&](const int* d) {
        try { t.put(d, sizeof(a), &copies, fail); } catch (const std::runtime_error&) { return true; }
        return false;
    };
    if (!fails(a)) return 1;              // nothing is held yet
    t.put(a, sizeof(a), &copies, copy);   // the failed copy left nothing behind
    t.put(a, sizeof(a), &copies, copy);   // held
    if (copies != 1 || fails(a)) return 2;
    t.put(a, sizeof(a), &other, copy);    // another order
    t.put(a, sizeof(int), &other, copy);  // another size
    if (copies != 3 || !fails(b)) return 3;
    t.put(a, sizeof(int), &other, copy);  // what was held before the failed copy is gone
    return copies == 4 ? 0 : 4;
}
"""


def test_failed_copies_are_not_remembered(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'csrc'}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
