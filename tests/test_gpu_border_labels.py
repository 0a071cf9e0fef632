"""Border extraction over the whole range of labels, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LOW = -2**31


@pytest.mark.parametrize("W,H", [(1, 1), (3, 5), (32, 32), (33, 65), (130, 97)])
@pytest.mark.parametrize("labels", [
    [LOW, LOW + 1, -9999, -9998], [LOW, -9998], [-9999, -9998, -9997, -9996, 0],
    [LOW, LOW + 1, -10000, -9999, -9998, -9997, -1, 0, 1, 2**31 - 2, 2**31 - 1]])
def test_border_of_any_label(cuda, oracle, W, H, labels):
    import torch
    from cageo_gb300 import api
    rng = np.random.default_rng(W + len(labels))
    lab = rng.choice(np.array(labels, np.int64), (H, W)).astype(np.int32)
    start = rng.integers(0, 4, (H, W)).astype(np.float32)
    counts = torch.from_numpy(start).to(cuda)
    api.border_accumulate(torch.from_numpy(lab).to(cuda), counts)
    assert np.array_equal(counts.cpu().numpy(), oracle.border_accumulate(lab, start))
