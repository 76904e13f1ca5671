"""map_pages brings an output array's pages in and, for a call that may yet fail, leaves its
contents as they are: fresh memory, pages of a file that are not in memory, arrays that start
and end inside a page.  Nothing outside the array changes in either form.
"""
import os
import shutil
import subprocess

import pytest
from conftest import ROOT

SRC = r"""
#include <fcntl.h>
#include <stdio.h>
#include <stdlib.h>
#include <vector>
#include "host_pages.h"
static size_t absent(void *p, size_t n) {
  const size_t page = sysconf(_SC_PAGESIZE);
  std::vector<unsigned char> in(n / page);
  mincore(p, n, in.data());
  size_t k = 0;
  for (unsigned char c : in) k += !(c & 1);
  return k;
}
int main(int argc, char **argv) {
  const size_t n = strtoull(argv[2], nullptr, 10), page = sysconf(_SC_PAGESIZE), len = n / page * page + 2 * page;
  const size_t off = strtoull(argv[3], nullptr, 10);
  const bool keep = atoi(argv[4]);
  // fresh memory
  char *a = (char *)mmap(0, len, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  const size_t before = absent(a, len);
  lmff::map_pages(a + off, n, keep);
  const size_t first = off / page, last = (off + n - 1) / page;
  if (absent(a + first * page, (last - first + 1) * page) != 0) return 1;
  if (before - absent(a, len) > last - first + 1) return 2;
  for (size_t k = 0; k < len; k++)
    if (a[k]) return 3;
  // a file's pages, dropped from memory where the file system does that
  int fd = open(argv[1], O_RDWR | O_CREAT | O_TRUNC, 0600);
  std::vector<char> v(len, 7);
  if (write(fd, v.data(), len) != (ssize_t)len) return 4;
  fsync(fd);
  posix_fadvise(fd, 0, len, POSIX_FADV_DONTNEED);
  char *f = (char *)mmap(0, len, PROT_READ | PROT_WRITE, MAP_SHARED, fd, 0);
  const size_t out = absent(f, len);
  lmff::map_pages(f + off, n, keep);
  for (size_t k = 0; k < len; k++)
    if (f[k] != 7 && (keep || k < off || k >= off + n)) return 5;
  printf("%zu\n", out);
  return 0;
}
"""


def test_contents_stay(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SRC)
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "lammps-lmff_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    for n, off in ((1, 0), (24, 4090), (4096, 0), (100_000, 8), (5 << 20, 24), ((9 << 20) + 8, 4088)):
        for keep in (1, 0):
            r = subprocess.run([str(exe), str(tmp_path / "f"), str(n), str(off), str(keep)], capture_output=True)
            assert r.returncode == 0, (n, off, keep, r.returncode)
