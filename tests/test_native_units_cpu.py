"""Native pieces that need no GPU, compiled on their own with fakes of the driver's calls."""
import shutil
import subprocess
import textwrap
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "csrc"
pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def _run(tmp_path, source):
    (tmp_path / "t.cpp").write_text(textwrap.dedent(source))
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{CSRC}", "-o", tmp_path / "t", tmp_path / "t.cpp"], check=True, timeout=120)
    return subprocess.run([tmp_path / "t"], check=True, timeout=60, capture_output=True, text=True).stdout.split()


def test_a_smaller_tile_never_takes_back_what_a_larger_one_was_granted(tmp_path):
    """Two threads ask at once; the one that wants more is slow to note that it was granted."""
    got = _run(tmp_path, """
        #include "kernels/smem_grant.h"
        #include <chrono>
        #include <cstdio>
        #include <thread>
        int main() {
          using namespace std::chrono_literals;
          SmemGrant grant;
          std::atomic<size_t> attribute{0};
          std::atomic<int> calls{0};
          auto set = [&](size_t bytes) {
            ++calls;
            attribute = bytes;
            if (bytes > 49000) std::this_thread::sleep_for(300ms);
            return 0;
          };
          std::thread large([&] { grant.ask(0, 50688, set); });
          while (attribute == 0) std::this_thread::yield();
          std::thread small([&] { grant.ask(0, 48576, set); });
          large.join();
          small.join();
          const int refused = grant.ask(0, 50688, set);
          std::printf("%zu %d %d ", attribute.load(), calls.load(), refused);
          // another device, a failure that is not noted, and a device beyond the table
          const int failed = grant.ask(1, 60000, [](size_t) { return 7; }), then = grant.ask(1, 60000, set), far = grant.ask(1000, 60000, set);
          std::printf("%d %d %d %d", failed, then, far, calls.load());
        }""")
    assert got == ["50688", "1", "0", "7", "0", "0", "3"]


def test_a_staging_buffer_that_cannot_be_had_is_not_asked_for_again(tmp_path):
    """The GPU has 8 MiB left: 16 are refused once, 4 and then 8 are had, what is larger stays refused."""
    got = _run(tmp_path, """
        #include "transport/staging_buffer.h"
        #include <cstdio>
        #include <initializer_list>
        int main() {
          kvx::StagingBuffer b;
          static char memory[2];
          int asked = 0, given = 0, back = 0;
          auto alloc = [&](size_t n) -> void* { ++asked; return n <= (8u << 20) ? &memory[given++] : nullptr; };
          auto release = [&](void*) { ++back; };
          auto step = [&](size_t mib) {
            const bool ok = b.reserve(mib << 20, alloc, release);
            std::printf("%d/%d ", static_cast<int>(ok), asked);
          };
          for (size_t mib : {16, 16, 32, 16, 4, 4, 16, 8, 2, 16}) step(mib);
          std::printf("%d %d", given, back);
          return b.data() == &memory[1] ? 0 : 1;
        }""")
    assert got == ["0/1", "0/1", "0/1", "0/1", "1/2", "1/2", "0/2", "1/3", "1/3", "0/3", "2", "1"]


def test_one_thread_at_a_time_looks_for_its_record(tmp_path):
    got = _run(tmp_path, """
        #include "core/own_look.h"
        #include <cstdio>
        #include <thread>
        #include <vector>
        using kvx::OwnLook;
        int main() {
          bool other = true, second = false;
          {
            OwnLook mine;
            std::thread([&] { OwnLook l; other = static_cast<bool>(l); }).join();
            OwnLook again;      // one that did not get it gives nothing back
            std::printf("%d %d %d ", static_cast<bool>(mine), other, static_cast<bool>(again));
          }
          std::thread([&] { OwnLook l; second = static_cast<bool>(l); }).join();
          std::atomic<int> inside{0}, most{0}, had{0};
          std::vector<std::thread> all;
          for (int t = 0; t < 8; ++t)
            all.emplace_back([&] {
              for (int i = 0; i < 2000; ++i) {
                OwnLook l;
                if (!l) continue;
                const int n = ++inside;
                if (n > most) most = n;
                ++had;
                OwnLook::pause();
                --inside;
              }
            });
          for (auto& t : all) t.join();
          std::printf("%d %d %d", second, most.load(), had.load() > 0);
        }""")
    assert got == ["1", "0", "0", "1", "1", "1"]
