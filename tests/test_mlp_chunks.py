"""The fused training passes at the edges of k_bwd_rows's chunk of 32 x 256 rows (a full chunk, a second chunk of one
residue group, three chunks) against the layer-by-layer passes, as in test_mlp_fused.py: the forward pass and dW
bit for bit, db to the rounding of a sum in another order."""
import pytest

from test_mlp_fused import test_fused_passes_match_layer_by_layer as compare


@pytest.mark.gpu
@pytest.mark.parametrize("act", ["gelu", "relu"])
@pytest.mark.parametrize("n", [8192, 8208, 20000])
def test_chunks_of_rows(n, act):
    compare(n, act)
