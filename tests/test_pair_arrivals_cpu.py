"""Arrivals that cross the CTAs of a pair name their scope.  An mbarrier arrival without one orders memory inside its
own CTA only, whichever CTA's barrier it is made on; the compiler accepts it and runs rarely show the difference, so
the sources are looked at: every arrival on a shared::cluster address is .release.cluster or .relaxed.cluster, and
the MMA warps' waits on barriers that the other CTA arrives on acquire at cluster scope."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dcvc_b200", "csrc")


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def test_arrivals_on_the_other_cta_name_their_scope():
    seen = 0
    for name, text in _sources():
        for m in re.finditer(r"mbarrier\.arrive([.\w:]*)\.shared::cluster", text):
            seen += 1
            assert m.group(1) in (".release.cluster", ".relaxed.cluster"), (name, m.group(0))
    assert seen > 0


def test_waits_for_the_other_cta_acquire_at_cluster_scope():
    text = dict(_sources())
    for name in ("dcb_sm100.cu", "quad_sm100.cu"):
        assert "if (!mbar_wait_warp<true>(bar, parity" in text[name], name
    gemm = text["gemm_sm100.cu"]
    assert "mbar_wait_warp<PAIR>(&tempty[acc]" in gemm and "mbar_wait_warp<PAIR>(&full[stage]" in gemm
    assert "mbar_test<PAIR>(&full[next]" in gemm
