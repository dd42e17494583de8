"""When look-back words are zeroed (csrc/vox_epochs.h), on the host: launches that use the words among
launches that use others (graph replays, whatever their pattern) never find a word of their own 24-bit
tag. Zeroing at exact multiples of the period would: a replay and a launch in turn step over every one
of them, and the tags repeat after 2^24 launches.
"""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(REPO, "wgpu-voxel-engine_gb300", "csrc")

CHECK = r"""
#include <cstdio>
#include <vector>
#include "vox_epochs.h"

// One word per launch size class, written by the launches that use it with their tag; `other`
// launches pass between two of them. Returns whether a launch met a word of its own tag.
static bool meets_own_tag(unsigned long long other, bool by_multiple) {
  vox::EpochWipe wipe;
  unsigned long long launches = 0;
  long word[2] = {-1, -1};  // a word that every launch writes, and one that only a rare one does
  for (unsigned k = 0; launches < (3ull << 24); ++k) {
    launches += other;
    const bool zero = by_multiple ? launches > 0 && (launches & (vox::kStateWipePeriod - 1)) == 0
                                  : wipe.due(launches);
    if (zero) word[0] = word[1] = -1;
    const long tag = (long)(launches & 0xFFFFFFull);
    ++launches;
    if (word[0] == tag || word[1] == tag) return true;
    word[0] = tag;
    if (k == 0) word[1] = tag;
  }
  return false;
}

int main() {
  const unsigned long long others[] = {0, 1, 2, 3, 7, 64, 1000003};
  for (unsigned long long o : others)
    if (meets_own_tag(o, false)) {
      std::printf("a tag repeats with %llu other launches between\n", o);
      return 1;
    }
  if (!meets_own_tag(1, true)) {
    std::printf("the multiples were not stepped over\n");
    return 1;
  }
  std::printf("ok\n");
  return 0;
}
"""


def test_words_are_zeroed_before_a_tag_repeats(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
