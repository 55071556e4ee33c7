"""Which evaluation's contact memory counts (memoryHolds in gdem_types.h), on the
host: the one before with the plain step, any that wrote with the coupled one,
also where the 32-bit count of evaluations has passed its largest value."""
import subprocess
import textwrap
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "pacific_b200" / "csrc"

PROGRAM = textwrap.dedent(r"""
    #include <climits>
    #include <cstdio>
    #include "gdem_types.h"
    using gdem::memoryHolds;
    int main() {
      int bad = 0;
      const unsigned starts[] = {1u, 511u, 4095u, (unsigned)INT_MAX - 4u, 0x80000005u, 0xF0000000u};
      for (unsigned s : starts)
        for (unsigned k = 0; k < 10; ++k) {
          const int now = (int)(s + k);
          if (memoryHolds(1, gdem::kNeverWritten, now) || memoryHolds(0, gdem::kNeverWritten, now)) ++bad;
          for (unsigned back = 0; back < 6; ++back) {
            const int e = (int)((unsigned)now - back);
            if (e == gdem::kNeverWritten) continue;
            if (memoryHolds(1, e, now) != (back == 1)) ++bad;
            if (!memoryHolds(0, e, now)) ++bad;
          }
        }
      std::printf("%d wrong\n", bad);
      return bad != 0;
    }
""")


def test_memory_of_any_evaluation(tmp_path):
    src = tmp_path / "holds.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "holds"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
