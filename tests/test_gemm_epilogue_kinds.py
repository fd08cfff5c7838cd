"""The epilogues of the CTA-pair kernel that are chosen on the host: a problem that wants column sums gets a form that leaves them."""

import os
import subprocess

import pytest

_CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "returnn_b200", "csrc")

_MAIN = r"""
#include "gemm_epilogue.cuh"
#include <stdio.h>
using namespace rbg;
void rb_set_error(const char*, ...) {}
bool rb_pdl_enabled() { return false; }
int main() {
  float sums[8], bias[4];
  for (int form = 0; form < 3; ++form)
    for (int drop = 0; drop < 2; ++drop)
      for (int wanted = 0; wanted < 2; ++wanted) {
        Params p = {};
        p.g = RbGemm();
        p.g.m = p.g.n = 256;
        p.tma_store = 1;
        if (form == 1) p.g.dact_z = bias, p.g.act = 2;
        if (form == 2) p.g.resid = bias;
        p.g.drop_p = drop ? 0.1f : 0.f;
        p.g.colsum = wanted ? sums : nullptr;
        const int k = epilogue_kind(p);
        printf("%d %d %d %d %d\n", form, drop, wanted, k, k == kEpiAny || k == kEpiDact || k == kEpiDactDrop);
      }
}
"""


def test_column_sums_have_an_epilogue_that_leaves_them(tmp_path):
    from returnn_b200.ops import build

    nvcc = build._nvcc()
    if not nvcc:
        pytest.skip("no compiler")
    (tmp_path / "main.cu").write_text(_MAIN)
    subprocess.run([nvcc] + [f for f in build.NVCC_FLAGS if f != "-O3"] + ["-I", _CSRC, "-o", str(tmp_path / "main"), str(tmp_path / "main.cu")], check=True)
    out = subprocess.run([str(tmp_path / "main")], check=True, stdout=subprocess.PIPE).stdout.decode().split("\n")
    rows = [tuple(map(int, line.split())) for line in out if line]
    assert len(rows) == 12
    for form, drop, wanted, kind, leaves in rows:
        # (form 0 without dropout has no column sums: rb_gemm_column_sums refuses it)
        assert leaves or not wanted or (form, drop) == (0, 0), (form, drop, kind)
    assert len({r[3] for r in rows if not r[2]}) == 6  # each has a form of its own, the generic one for dropout alone
