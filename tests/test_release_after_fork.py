"""Releasing a buffer takes no lock of the library's own: a child forked while
other threads release buffers can release its own, as with any malloc'd memory.

A C caller of the library does it (threads of an interpreter release too
seldom to be caught at it); no GPU is needed, the buffers are malloc'd as the
library's results are."""

import os
import shutil
import subprocess

import pytest

from metalmom_b200._native import LIB_PATH

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <pthread.h>
#include <stdio.h>
#include <stdlib.h>
#include <sys/wait.h>
#include <unistd.h>
#include "metalmom.h"
static volatile int stop;
static void *work(void *p) {
  while (!stop) {
    MMBuffer b = {0};
    b.data = malloc(64);
    mm_buffer_free(&b);
  }
  return p;
}
int main(void) {
  pthread_t t[4];
  int bad = 0;
  for (int i = 0; i < 4; i++) pthread_create(&t[i], 0, work, 0);
  for (int i = 0; i < 200 && !bad; i++) {
    MMBuffer mine = {0};
    mine.data = malloc(64);
    pid_t pid = fork();
    if (pid == 0) {
      alarm(10); /* ends a child that waits for a lock nobody will release */
      mm_buffer_free(&mine);
      _exit(mine.data ? 3 : 0);
    }
    int status = 0;
    if (waitpid(pid, &status, 0) != pid || status != 0) bad = printf("fork %d: status %d\n", i, status);
    mm_buffer_free(&mine);
  }
  stop = 1;
  for (int i = 0; i < 4; i++) pthread_join(t[i], 0);
  return bad ? 1 : 0;
}
"""


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc for the C caller")
def test_a_forked_child_releases_buffers(tmp_path):
    src, exe = tmp_path / "fork.c", tmp_path / "fork"
    src.write_text(PROGRAM)
    subprocess.check_call(["gcc", "-O1", "-o", str(exe), str(src), "-I", os.path.join(ROOT, "include"), LIB_PATH,
                           "-Wl,-rpath," + os.path.dirname(LIB_PATH), "-Wl,--allow-shlib-undefined", "-lpthread"])
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
