"""A stand-in for cudaLaunchCooperativeKernel, compiled and preloaded into a child
process: it counts the launches by kernel name and, on request, refuses them as
the runtime refuses a grid that cannot be co-resident, or leaves out the last
block of the grid.  Beside it one for cudaMalloc that adds up the bytes."""
import os
import subprocess
import sys
import textwrap

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))

SRC = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <string.h>
typedef struct { unsigned x, y, z; } dim;
typedef int (*launch_t)(const void*, dim, dim, void**, unsigned long, void*);
typedef int (*name_t)(const char**, const void*);
static int refuse_, drop_;
static unsigned long bytes_;
unsigned long malloc_bytes(void) { return bytes_; }
int cudaMalloc(void** p, unsigned long n) {
  static int (*next)(void**, unsigned long);
  if (!next) next = (int (*)(void**, unsigned long))dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaMalloc");
  bytes_ += n;
  return next(p, n);
}
static char names_[1 << 20];
void coop_refuse(int on) { refuse_ = on; }
void coop_drop(int on) { drop_ = on; }
void coop_clear(void) { names_[0] = 0; }
const char* coop_names(void) { return names_; }
int cudaLaunchCooperativeKernel(const void* f, dim g, dim b, void** args, unsigned long smem, void* stream) {
  static launch_t next;
  static name_t name;
  if (!next) {
    void* rt = dlopen("libcudart.so.13", RTLD_LAZY); /* the one the library has loaded */
    next = (launch_t)dlsym(rt, "cudaLaunchCooperativeKernel");
    name = (name_t)dlsym(rt, "cudaFuncGetName");
  }
  if (refuse_) return 720; /* cudaErrorCooperativeLaunchTooLarge */
  const char* n = "?";
  if (name) name(&n, f);
  if (strlen(names_) + strlen(n) + 2 < sizeof names_) {
    strcat(names_, n);
    strcat(names_, "\n");
  }
  if (drop_ && g.x > 1) g.x -= 1;
  return next(f, g, b, args, smem, stream);
}
"""

HEAD = """
import ctypes as C, os, sys
sys.path.insert(0, {root!r})
import numpy as np
lib = C.CDLL({so!r})
lib.coop_names.restype = C.c_char_p
lib.malloc_bytes.restype = C.c_ulong
def launched():
    names = lib.coop_names().decode().split()
    lib.coop_clear()
    return names
"""


def run(tmp_path, head, code, timeout=300):
    """head + code in a child process with the stand-in preloaded; its output."""
    src, so = tmp_path / "coop.c", tmp_path / "coop.so"
    src.write_text(SRC)
    subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(src), "-o", str(so), "-ldl"], check=True)
    env = dict(os.environ, LD_PRELOAD=str(so))
    r = subprocess.run([sys.executable, "-c", HEAD.format(root=ROOT, so=str(so)) + head + textwrap.dedent(code)], env=env,
                       capture_output=True, text=True, timeout=timeout, cwd=ROOT)
    assert r.returncode == 0, r.stdout + r.stderr
    return r.stdout
