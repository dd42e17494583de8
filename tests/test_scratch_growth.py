"""Growth of a context's per-chunk scratch (csrc/vox_scratch.h) on the host, over an allocator that runs
out of memory: how much a small batch takes, what is kept where the face lists' slots do not fit, and
that a size without room is asked for once.
"""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "wgpu-voxel-engine_gb300", "csrc")

CHECK = r"""
#include <cstdio>
#include <cstdlib>
#include <map>
#include "vox_scratch.h"

struct Memory {
  size_t room, used = 0;
  int other = 0;  // an error of another kind, given once
  long calls = 0, released = 0, next = 1;
  std::map<void*, size_t> held;
  int alloc(size_t bytes, void** p) {
    ++calls;
    if (other) { const int e = other; other = 0; return e; }
    if (bytes > room - used) return 2;
    *p = (void*)(next++ * 16);
    held[*p] = bytes;
    used += bytes;
    return 0;
  }
  void release(void* p) {
    if (!held.count(p)) { std::printf("not held\n"); std::exit(1); }
    ++released;
    used -= held[p];
    held.erase(p);
  }
};

constexpr size_t kList = 128, kSpill = 59, kFloor = 1024 * kSpill;

static int grow(Memory& m, vox::ScratchBuffer& b, size_t n, bool& lists, size_t list = kList) {
  return vox::grow_scratch(b, n, list, kSpill, kFloor, lists, 2,
                           [&](size_t bytes, void** p) { return m.alloc(bytes, p); }, [&](void* p) { m.release(p); });
}
#define CHECK_THAT(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
  bool lists;
  {  // a small batch takes the floor, not 1024 list slots; a large one what it needs
    Memory m{1u << 30};
    vox::ScratchBuffer b;
    CHECK_THAT(grow(m, b, 1, lists = true) == 0 && lists && b.bytes == kFloor);
    CHECK_THAT(grow(m, b, kFloor / kList, lists = true) == 0 && m.calls == 1);
    CHECK_THAT(grow(m, b, 2000, lists = true) == 0 && lists && b.bytes == 2000 * kList && m.used == b.bytes);
    CHECK_THAT(grow(m, b, 3000, lists = false) == 0 && !lists && m.calls == 2);  // fits: 3000 * 59
  }
  {  // lists do not fit: the buffer at hand serves, is kept, and the size is asked for once
    Memory m{200000};
    vox::ScratchBuffer b;
    CHECK_THAT(grow(m, b, 2000, lists = false) == 0 && b.bytes == 2000 * kSpill);
    void* kept = b.data;
    for (int k = 0; k < 5; ++k) {
      lists = true;
      CHECK_THAT(grow(m, b, 2000, lists) == 0 && !lists && b.data == kept);
    }
    CHECK_THAT(m.calls == 2 && m.released == 0);
    CHECK_THAT(grow(m, b, 600, lists = true) == 0 && lists && b.data == kept);  // a smaller one still lists
    // a larger batch does not ask for lists again
    CHECK_THAT(grow(m, b, 3000, lists = true) == 0 && !lists && b.bytes == 3000 * kSpill);
    CHECK_THAT(m.calls == 4 && m.used == b.bytes);  // (with the old buffer first, then in its place)
  }
  {  // no buffer yet: lists, then the smaller slots
    Memory m{150000};
    vox::ScratchBuffer b;
    CHECK_THAT(grow(m, b, 2000, lists = true) == 0 && !lists && b.bytes == 2000 * kSpill && m.used == b.bytes);
    const long calls = m.calls;
    CHECK_THAT(grow(m, b, 2000, lists = true) == 0 && !lists && m.calls == calls);
  }
  {  // room for the new buffer only without the old one
    Memory m{300000};
    vox::ScratchBuffer b;
    CHECK_THAT(grow(m, b, 1500, lists = true) == 0 && lists);
    CHECK_THAT(grow(m, b, 2300, lists = true) == 0 && !lists && b.bytes == 1500 * kList);  // serves 2300 * 59
    CHECK_THAT(grow(m, b, 4000, lists = false) == 0 && b.bytes == 4000 * kSpill && m.used == b.bytes);
  }
  {  // no room at all, and errors of another kind: reported, the latter with nothing given back
    Memory m{100000};
    vox::ScratchBuffer b;
    CHECK_THAT(grow(m, b, 10, lists = true) == 0 && lists);
    void* kept = b.data;
    m.other = 7;
    CHECK_THAT(grow(m, b, 1700, lists = true) == 7 && b.data == kept);
    CHECK_THAT(grow(m, b, 9000, lists = true) == 2 && b.data == nullptr && b.bytes == 0 && m.used == 0);
    CHECK_THAT(grow(m, b, 10, lists = true) == 0 && lists && b.bytes == kFloor);
  }
  {  // one size of slots: no choice to make
    Memory m{100000};
    vox::ScratchBuffer b;
    CHECK_THAT(grow(m, b, 1600, lists = true, kSpill) == 0 && lists);
    CHECK_THAT(grow(m, b, 1800, lists = true, kSpill) == 2 && lists);
  }
  std::printf("ok\n");
  return 0;
}
"""


def test_scratch_growth(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
