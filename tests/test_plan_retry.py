"""A plan whose device memory could not be had leaves nothing behind: the
call after a failed one fails again or builds all of it.  Run without a
device, where every allocation fails, through the library's internal
functions (a small program, compiled here against its header)."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PROGRAM = r"""
#include <cstdio>
#include <cstring>
#include <initializer_list>

#include "qd_internal.hpp"

int main(int argc, char** argv) {
  qd_layout* L = nullptr;
  if (argc < 2 || qd_layout_create(2, 4, nullptr, QD_HOST_ONLY, &L)) return 2;
  for (int call = 0; call < 3; ++call) {
    int rc = -1;
    if (!strcmp(argv[1], "ph_gen")) rc = qd::prepare_ph_gen(L);
    if (!strcmp(argv[1], "onebody")) rc = qd::prepare_onebody(L);
    if (!strcmp(argv[1], "programs")) {
      rc = qd::build_programs(L);
      size_t n = 0;
      for (qd::GemmProgram* P : {&L->prog_ladder, &L->prog_ladder_gen, &L->prog_221, &L->prog_111, &L->prog_pandya})
        n += P->probs.size() + P->segs.size() + (P->d_probs || P->d_segs);
      printf("%d %d %zu\n", rc != QD_OK, (int)L->programs_built, n);
      continue;
    }
    printf("%d %d %zu\n", rc != QD_OK, L->ph_gen || L->onebody, L->dev_allocs.size());
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("plans")
    src, exe = d / "plans.cpp", d / "plans"
    src.write_text(PROGRAM)
    lib = os.path.join(ROOT, "qd_imsrg_b200")
    subprocess.check_call(["g++", "-std=c++17", "-O0", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(lib, "csrc"), "-I", "/usr/local/cuda/include", str(src), "-o", str(exe),
                           "-L", lib, "-l:libqdimsrg.so", "-Wl,-rpath," + lib])
    return str(exe)


def calls(program, what):
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    out = subprocess.run([program, what], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    return [tuple(int(x) for x in line.split()) for line in out.stdout.splitlines()]


@pytest.mark.parametrize("plan", ["ph_gen", "onebody", "programs"])
def test_failed_plan_is_not_kept(program, plan):
    # every call fails, no plan and no memory is kept
    assert calls(program, plan) == [(1, 0, 0)] * 3
