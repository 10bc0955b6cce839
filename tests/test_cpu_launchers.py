"""Launchers that refuse a call before they launch anything (csrc/kernels.cuh), called from a small host program: no GPU
takes part."""
import os
import subprocess

import hdog

CSRC = os.path.join(hdog._PKG, "csrc")


def run(tmp_path, body):
    src, exe = str(tmp_path / "t.cu"), str(tmp_path / "t")
    with open(src, "w") as f:
        f.write('#include <cstdio>\n#include "kernels.cuh"\nusing namespace hdog;\nint main() {\n%s\n}\n' % body)
    out = os.path.dirname(hdog.LIB_PATH)
    r = subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-I", CSRC, "-I",
                        os.path.join(os.path.dirname(hdog._PKG), "include"), src, "-o", exe, "-L" + out,
                        "-lhdog", "-Xlinker", "-rpath," + out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    return r.returncode, r.stdout


def test_a_volume_that_no_tensor_map_takes_is_refused(tmp_path):
    """The DoG volume off its 16 bytes (and, without a driver, no encoder at all): a status, no launch."""
    rc, out = run(tmp_path, """
  DogTaps T{};
  float *off = reinterpret_cast<float *>(4);
  const int rc = launch_dog_hess(nullptr, 1, 64, 64, 64, 8, T, nullptr, nullptr, nullptr, off, nullptr, nullptr, nullptr,
                                 nullptr, nullptr, LaunchShape{}, nullptr, 1 << 16, nullptr);
  printf("%d\\n", rc);
  return rc == HDOG_ERR_CUDA ? 0 : 1;""")
    assert rc == 0, (rc, out)


def test_a_list_of_more_ranges_than_it_holds_is_refused(tmp_path):
    """One range too many leaves the others as they are and the list refused."""
    rc, out = run(tmp_path, """
  struct { ClearList z; uint32_t guard[64]; } s;
  for (uint32_t &g : s.guard) g = 7;
  uint32_t words[4];
  for (int i = 0; i < ClearList::kMax; i++) s.z.add(words, 4 * (i + 1));
  const ClearList full = s.z;
  if (full.over) return 2;
  s.z.add(words + 1, 16);
  bool same = s.z.count == full.count;
  for (int i = 0; i < ClearList::kMax; i++) same &= s.z.p[i] == full.p[i] && s.z.n[i] == i + 1;
  for (uint32_t g : s.guard) same &= g == 7;
  return same && s.z.over && clear_async(s.z, nullptr) == HDOG_ERR_CAPACITY ? 0 : 1;""")
    assert rc == 0, (rc, out)
