"""Keys of the captured graphs: two operators whose members are equal have the same key whatever lies in the
bytes between and behind the members, and every member is part of it."""
import os
import subprocess

import pytest

from conftest import ROOT
from h2_b200 import build

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include <new>
#include "h2g_internal.cuh"
using namespace h2g;

template <typename T>
static void fill(OpParams<T>& op) {
  op.g.MX = 1; op.g.MY = 2; op.g.MZ = 3; op.g.NX = 4; op.g.NY = 5; op.g.NZ = 6; op.g.HP = 7; op.g.HI = 8; op.g.HN = 9;
  op.g.plane = 10; op.g.n = 11;
  op.key = nullptr; op.tx = op.ty = op.tz = op.conv = op.rc = op.dzk = op.ddv = op.tq = op.ctab = nullptr;
  op.nkey = nullptr; op.cls = nullptr;
  op.czm = op.czp = op.dx0 = op.dy0 = op.ddt = T(1);
  op.P = 12; op.steady = 1; op.cls_dd = 1;
}
template <typename T>
static int check() {
  alignas(16) static unsigned char a[sizeof(OpParams<T>)], b[sizeof(OpParams<T>)];
  memset(a, 0x00, sizeof a);
  memset(b, 0xff, sizeof b);
  auto& x = *reinterpret_cast<OpParams<T>*>(a);
  auto& y = *reinterpret_cast<OpParams<T>*>(b);
  fill(x);
  fill(y);
  std::vector<unsigned char> ka, kb;
  append_members(ka, x);
  append_members(kb, y);
  if (ka != kb) return 1;
  // a byte of the struct changes the key exactly if it belongs to a member, and a member is every byte that
  // filling the members defined
  for (size_t q = 0; q < sizeof a; ++q) {
    const bool member = a[q] == b[q];
    a[q] ^= 1;
    std::vector<unsigned char> kc;
    append_members(kc, x);
    a[q] ^= 1;
    if ((kc != ka) != member) return 2;
  }
  return 0;
}
int main() { printf("%d %d", check<double>(), check<float>()); }
"""


def test_key_is_the_members(tmp_path):
    src, exe = tmp_path / "key.cu", tmp_path / "key"
    src.write_text(SOURCE)
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("no nvcc")
    subprocess.run([nvcc, "-std=c++17", "-O0", "-I", os.path.join(ROOT, "h2_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True, capture_output=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout == "0 0"


def test_no_key_is_copied_from_a_struct():
    """The solver makes its keys with append_members and append_bytes alone."""
    text = open(os.path.join(ROOT, "h2_b200", "csrc", "h2g_solver.cu")).read()
    for name in ("signature", "sign_resident"):
        body = text[text.index(f" {name}("):]
        body = body[:body.index("\n}")]
        assert "memcpy" not in body and "sizeof" not in body and "append_bytes" in body, name
    assert "sizeof op" not in text
