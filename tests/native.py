"""Small C++ programs over libaqua's own structures (csrc/internal.h), for tests
that must see or set what the C ABI does not show: compiled with g++ and linked
to the library under test."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT

PRELUDE = r"""
#include <cstdio>
#include <cstring>
#include <vector>
#include "internal.h"

#define CHECK(c)                                                 \
    do {                                                         \
        if (!(c)) {                                              \
            printf("line %d: %s\n", __LINE__, #c);               \
            return 1;                                            \
        }                                                        \
    } while (0)

// The next device allocation of the context fails, and no later one.
static inline void fail_next_alloc(aqua_ctx* ctx) {
    ctx->fail_alloc_after = ~0ull;
    ctx->alloc_count = ~0ull - 1;
}
"""


def run(tmp_path, program: str) -> str:
    gxx, cuda = shutil.which("g++"), os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(PRELUDE + program)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I" + os.path.join(PKG, "csrc"), "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"), str(src), "-o", str(exe), "-L" + PKG, "-laqua",
                    "-L" + os.path.join(cuda, "lib64"), "-lcudart", "-Wl,-rpath," + PKG,
                    "-Wl,-rpath," + os.path.join(cuda, "lib64")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout + out.stderr
    return out.stdout
