"""The kept answers of occupancy queries (csrc/ag_occupancy.h), compiled with the thread sanitizer: launches with several
row lengths in turn ask once per length, from any number of threads, and no answer is given for another length's question."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "ag_occupancy.h"

static AgOccupancy known;
static std::atomic<int> asked{0}, wrong{0};

static int right(int threads, size_t smem) { return 1 + (int)((threads / 32 + smem / 1024) % 16); }

static void launch(int threads, size_t smem) {
  const int occ = known.get(threads, smem, [&] { asked++; return right(threads, smem); });
  if (occ != right(threads, smem)) wrong++;
}

int main(int argc, char** argv) {
  const int keys = std::atoi(argv[1]), workers = std::atoi(argv[2]);
  if (known.get(256, 0, [] { return -1; }) != -1) return 2;   // an error is handed through and not kept
  std::vector<std::thread> all;
  for (int w = 0; w < workers; ++w)
    all.emplace_back([=] { for (int i = 0; i < 4000; ++i) launch(32 * (1 + (i + w) % 3 % keys), 1024 * ((i + w) % keys)); });
  for (auto& t : all) t.join();
  std::printf("%d %d\n", asked.load(), wrong.load());
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    where = tmp_path_factory.mktemp("occupancy")
    src, exe = where / "main.cpp", where / "main"
    src.write_text("#include <cstdlib>\n" + PROGRAM)
    cmd = [gxx, "-std=c++17", "-O1", "-g", "-pthread", "-I", os.path.join(ROOT, "autograd_b200", "csrc"), str(src), "-o", str(exe)]
    probe = subprocess.run(cmd + ["-fsanitize=thread"], capture_output=True, text=True)
    if probe.returncode != 0:      # no sanitizer runtime: the counts are checked all the same
        subprocess.run(cmd, check=True)
    return str(exe)


@pytest.mark.parametrize("keys,workers", [(1, 1), (2, 1), (2, 8), (7, 8), (23, 8)])
def test_answers_are_right_and_kept(program, keys, workers):
    r = subprocess.run([program, str(keys), str(workers)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
    asked, wrong = map(int, r.stdout.split())
    assert wrong == 0
    shapes = len({(i % 3 % keys, i % keys) for i in range(3 * keys)})
    if shapes <= 8:
        assert asked <= shapes * workers     # threads that miss together ask together
