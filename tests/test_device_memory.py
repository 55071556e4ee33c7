"""Bookkeeping of a system's device memory (gdem_memory.h) on the host, with an
arena in the device's place: arrays never overlap, nothing is given back while
an array lives in it, everything is given back once at the end.

The sequence is a system's: arrays that stay, then lists out of the same blocks
that may be given back when they outgrow them (for some sizes such a list opens
a block of its own, and the arrays that follow share it), for every capacity
from 1 to 20,000 particles, with blocks that cannot be had among them."""
import subprocess
import textwrap
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "pacific_b200" / "csrc"

PROGRAM = textwrap.dedent(r"""
    #include <cstdint>
    #include <cstdio>
    #include <cstdlib>
    #include <map>
    #include "gdem_memory.h"
    typedef std::uintptr_t U;
    static std::map<U, std::size_t> live;      // what the device has handed out
    static U at = 1 << 20;
    static std::size_t limit = ~std::size_t(0);
    static int bad = 0;
    static void* take(std::size_t n) {
      if (n > limit) return nullptr;
      at = (at + 511) & ~U(511);
      live[at] = n;
      void* p = reinterpret_cast<void*>(at);
      at += n;
      return p;
    }
    static void give(void* p) { if (!live.erase(reinterpret_cast<U>(p))) ++bad; }
    static bool inside(U p, std::size_t n) {
      auto it = live.upper_bound(p);
      if (it == live.begin()) return false;
      --it;
      return p >= it->first && p + n <= it->first + it->second;
    }
    int main() {
      for (std::size_t cap = 1; cap <= 20000; cap += cap < 400 ? 1 : 37) {
        limit = cap % 11 == 0 ? 64 * cap : ~std::size_t(0);
        std::map<U, std::size_t> arrays;
        {
          gdem::DeviceMemory m(take, give);
          auto add = [&](void* p, std::size_t n) {
            const U u = reinterpret_cast<U>(p);
            if (!p) return;
            if (u % 256) ++bad;
            auto it = arrays.lower_bound(u);
            if (it != arrays.end() && u + n > it->first) ++bad;
            if (it != arrays.begin() && (--it, it->first + it->second > u)) ++bad;
            arrays[u] = n;
          };
          auto shared = [&](std::size_t n) {
            // (small blocks, which some arrays exceed, and large ones)
            void* p = m.shared(n, cap % 2 ? 1 << 18 : std::max((cap + 64) * 4096, m.sharedTotal()));
            add(p, n);
            return p;
          };
          auto back = [&](void* p) {
            if (!p) return;
            m.giveBack(p);
            arrays.erase(reinterpret_cast<U>(p));
          };
          for (int k = 0; k < 30; ++k) shared((k % 5 + 1) * 8 * cap);
          void* cells = m.own(4 * cap + 4096);
          add(cells, 4 * cap + 4096);
          void* pairs = shared((16 * cap + 4096) * (cap % 3 ? 112 : 64));
          for (int k = 0; k < 6; ++k) shared(16 * cap);
          void* walls = shared(cap * 6 * 180);
          for (int k = 0; k < 6; ++k) shared(k % 2 ? 176 * cap : 8);
          for (int round = 0; round < 3; ++round) {
            back(pairs);
            add(pairs = m.own((24 * cap + 4096) << round), (24 * cap + 4096) << round);
            back(walls);
            add(walls = m.own((cap * 9) << round), (cap * 9) << round);
            back(cells);
            add(cells = m.own(8 * cap), 8 * cap);
            for (auto const& a : arrays)
              if (!inside(a.first, a.second) && bad++ < 5)
                std::printf("capacity %zu: an array of %zu bytes was given back\n", cap, a.second);
          }
        }
        if (!live.empty()) ++bad;
        live.clear();
      }
      std::printf("%d faults\n", bad);
      return bad != 0;
    }
""")


def test_nothing_live_is_given_back(tmp_path):
    src = tmp_path / "memory.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "memory"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
