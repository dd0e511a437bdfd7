"""The helper threads of host copies and a fork: a child of a process whose helpers are waiting
runs its own copies without them and ends normally, through exit() as well."""
import os
import subprocess

from conftest import PKG

PROGRAM = r"""
#include <signal.h>
#include <stdio.h>
#include <stdlib.h>
#include <sys/wait.h>
#include <unistd.h>
#include <atomic>
#include "hostpool.h"

static int sum() {
  std::atomic<int> s{0};
  dmm::pool_run(8, [&](int i) { s += i; });
  return s.load();
}

int main() {
  if (sum() != 28) return 2;
  usleep(20000);  // the helpers are asleep
  fflush(stdout);
  const pid_t p = fork();
  if (p == 0) exit(sum() == 28 ? 7 : 8);
  for (int k = 0; k < 100; k++) {
    int st;
    if (waitpid(p, &st, WNOHANG) == p)
      return WIFEXITED(st) && WEXITSTATUS(st) == 7 && sum() == 28 ? 0 : 3;
    usleep(100000);
  }
  kill(p, SIGKILL);
  waitpid(p, nullptr, 0);
  return 4;  // the child did not end
}
"""


def test_forked_child_ends(tmp_path):
    src = tmp_path / "fork.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "fork")
    csrc = os.path.join(PKG, "csrc")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-I", csrc, "-I", "/usr/local/cuda/include",
                    str(src), os.path.join(csrc, "hostpool.cpp"), os.path.join(csrc, "devmem.cpp"),
                    "-o", exe, "-L", "/usr/local/cuda/lib64", "-lcudart_static", "-lpthread",
                    "-ldl", "-lrt"], check=True, timeout=300)
    r = subprocess.run([exe], timeout=60)
    assert r.returncode == 0
