"""Indices near the end of lists and fields of 2^31 - 2 entries, the most that
ddinit accepts: threads of a last block beyond the end must neither wrap to a
negative index nor pass for one inside.  The helpers that the kernels use
(ddc_internal.h) are compiled for the host; the loops that walk such lists are
read from the sources (a counter from zero, never the index itself plus the
stride)."""
import glob
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "ddpcm_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "ddc_internal.h"
int main() {
  const int top = 2147483646, q0 = top - 70;  // a last list of 70 entries
  for (int k : {0, 69, 70, 127, 255, 100000}) std::printf("%d ", ddc::list_entry(q0, top, k));
  // 2^31 - 2 points, blocks of 256 threads and two steps: the last block
  const unsigned np = 2147483646u, block = (np - 1) / 512;
  int inside = 0, wrapped = 0;
  for (unsigned i = 0; i < 2; ++i)
    for (unsigned t = 0; t < 256; ++t) {
      const unsigned p = ddc::step_point(block, 2, i, 256, t);
      inside += p < np;
      wrapped += p < block * 512u;
    }
  std::printf("%d %d\n", inside, wrapped);
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="g++ not available")
def test_helpers_at_the_end(tmp_path):
    src, exe = tmp_path / "i.cpp", tmp_path / "i"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-fsanitize=signed-integer-overflow",
                    "-fno-sanitize-recover", "-I", CSRC, "-I", "/usr/local/cuda/include",
                    "-o", exe, src], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    top = 2147483646
    assert [int(v) for v in out[:6]] == [top - 70] + [top - 1] * 5
    inside, wrapped = int(out[6]), int(out[7])
    assert inside == top - (top - 1) // 512 * 512 and wrapped == 0


def test_no_loop_steps_a_list_index():
    """`for (int q = <list start> + thread; q < end; q += stride)` overflows in
    the last list when fewer than `stride` indices are left."""
    lists = r"(ls_ptr|pn_ptr|q0|\ba)\b"
    for f in glob.glob(os.path.join(CSRC, "*.cu")):
        for start in re.findall(r"for \(int \w+ = ([^;]*(?:threadIdx\.x|lane|tid));", open(f).read()):
            assert not re.search(lists, start), (os.path.basename(f), start)


def test_kernels_use_the_helpers():
    text = {os.path.basename(f): open(f).read() for f in glob.glob(os.path.join(CSRC, "*.cu"))}
    assert "list_entry(q0, q1, entry(k, p))" in text["ddc_lxs.cu"]
    gather = text["ddc_kernels.cu"].split("k_lx_gather(")[1].split("gather_launch(")[0]
    assert gather.count("step_point(") == 2 and "blockIdx.x *" not in gather
