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
