"""Runs a script with some CUDA runtime calls of the library seen, or refused,
on the host: a preloaded object stands in front of them.  FAKE_HOST_MAX=n
refuses page-locked allocations above n bytes, FAKE_NO_TEXTURE=1 texture
objects.  In the script, calls() gives page-locked bytes held, texture objects
made, and the order of stream waits ("S") and texture releases ("T")."""
import os
import subprocess
import sys

from conftest import PKG_ROOT, ROOT

SRC = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>
static void* real(const char* name) {
  void* h = dlopen("libcudart.so.13", RTLD_LAZY | RTLD_NOLOAD);
  return h ? dlsym(h, name) : NULL;
}
static struct { void* p; size_t n; } held[4096];
static long bytes, textures;
static char order[4096];
static void note(char c) {
  size_t n = strlen(order);
  if (n + 1 < sizeof order) order[n] = c;
}
long fake_bytes(void) { return bytes; }
long fake_textures(void) { return textures; }
const char* fake_order(void) { return order; }
int cudaHostAlloc(void** p, size_t n, unsigned flags) {
  const char* max = getenv("FAKE_HOST_MAX");
  if (max && n > (size_t)atol(max)) { *p = NULL; return 2; }
  int e = ((int (*)(void**, size_t, unsigned))real("cudaHostAlloc"))(p, n, flags);
  for (int k = 0; e == 0 && k < 4096; k++)
    if (!held[k].p) { held[k].p = *p; held[k].n = n; bytes += (long)n; break; }
  return e;
}
int cudaFreeHost(void* p) {
  for (int k = 0; p && k < 4096; k++)
    if (held[k].p == p) { bytes -= (long)held[k].n; held[k].p = NULL; break; }
  return ((int (*)(void*))real("cudaFreeHost"))(p);
}
int cudaCreateTextureObject(unsigned long long* o, const void* r, const void* t, const void* v) {
  if (getenv("FAKE_NO_TEXTURE")) return 2;
  textures++;
  return ((int (*)(unsigned long long*, const void*, const void*, const void*))real("cudaCreateTextureObject"))(o, r, t, v);
}
int cudaDestroyTextureObject(unsigned long long o) {
  note('T');
  return ((int (*)(unsigned long long))real("cudaDestroyTextureObject"))(o);
}
int cudaStreamSynchronize(void* s) {
  note('S');
  return ((int (*)(void*))real("cudaStreamSynchronize"))(s);
}
"""

HEAD = """
import ctypes, hashlib, sys
sys.path[:0] = %r
import numpy as np
from eleven import _abi as A, _lib, scenes
fake = ctypes.CDLL(None)
fake.fake_bytes.restype = fake.fake_textures.restype = ctypes.c_long
fake.fake_order.restype = ctypes.c_char_p
def calls():
    return fake.fake_bytes(), fake.fake_textures(), fake.fake_order().decode()
def digest(*arrays):
    return hashlib.sha256(b"".join(np.ascontiguousarray(a).tobytes() for a in arrays)).hexdigest()
"""


def run(tmp_path, script, **env):
    """What the script prints."""
    so = tmp_path / "calls.so"
    if not so.exists():
        src = tmp_path / "calls.c"
        src.write_text(SRC)
        subprocess.run(["gcc", "-O1", "-shared", "-fPIC", str(src), "-o", str(so), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", HEAD % [PKG_ROOT, os.path.join(ROOT, "tests")] + script],
                       env=dict(os.environ, LD_PRELOAD=str(so), **env), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout.strip()
