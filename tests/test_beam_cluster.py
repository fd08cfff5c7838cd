"""The ranking's form in one kernel is taken only where the device says that it can place the clusters; where it cannot be asked, two kernels run."""

import pytest
import torch


@pytest.mark.parametrize("beam", [1, 8, 9, 16, 17])
def test_clusters_are_asked_for(beam):
    from returnn_b200.ops import _lib, seq_ops

    if _lib.get_lib() is None:
        pytest.skip("kernel library not built")
    fits = bool(_lib.bind("rb200_beam_topk_cluster_fits", [seq_ops._i32])(beam))
    assert fits == (torch.cuda.is_available() and beam <= 16)
    assert seq_ops._beam_cluster_fits(0, beam) == fits and not seq_ops._beam_cluster_fits(torch.cuda.device_count(), beam)


@pytest.mark.parametrize("B,beam,V,item,one", [
    (1, 12, 10001, 2, True), (64, 1, 32000, 2, True), (64, 4, 32000, 2, False), (64, 4, 1001, 2, True), (12, 8, 32000, 2, True), (16, 8, 32000, 2, False),
    (8, 8, 1001, 2, True), (16, 8, 1001, 2, False), (16, 8, 1001, 4, True), (8, 12, 1001, 2, False), (24, 12, 10001, 2, False), (4, 16, 32000, 2, True), (4, 16, 5001, 2, False),
    (8, 16, 10001, 2, False), (32, 16, 1001, 4, False), (1, 17, 100, 2, False)])
def test_form_by_size(B, beam, V, item, one):
    """both sides of the borders that were measured"""
    from returnn_b200.ops import seq_ops

    assert seq_ops._beam_one_kernel(B, beam, V, item) == one
