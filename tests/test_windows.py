"""When galic_optimize_reps runs the orbits of two windows at once (galic_b200/csrc/windows.h), on the CPU."""
import os
import subprocess

from conftest import ROOT

SRC = r'''
#include <cstdio>
#include <initializer_list>
#include "windows.h"
int main()
{
  // a call of one window has no second one to run beside it and makes no stream for it
  for(int largest : {1, 4096, 4097, 100000}) std::printf("%d", windows_paired(1, largest));
  for(int largest : {1, 4096, 4097, 100000}) std::printf("%d", windows_paired(2, largest));
  for(int largest : {4096, 4097}) std::printf("%d", windows_paired(7, largest));
}
'''


def test_only_calls_of_several_small_windows_pair(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "galic_b200", "csrc"), str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")], check=True, capture_output=True).stdout == b"0000110010"
