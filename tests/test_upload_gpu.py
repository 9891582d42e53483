"""Host arrays uploaded through one pinned buffer keep their shapes and types."""
import numpy as np
import pytest
import torch

from pot_gb300._arrays import upload

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.int32, np.int64, np.uint8, np.int16, np.bool_])
def test_upload_keeps_shape_and_type(cuda, dtype):
    x = (np.arange(6).reshape(2, 3) % 2).astype(dtype)
    got = upload(cuda, [x, x.T, x[:, :0], x[0, 0]])
    for t, w in zip(got, [x, x.T, x[:, :0], x[0, 0]]):
        w = np.asarray(w)
        assert t.is_cuda and tuple(t.shape) == w.shape and t.dtype == torch.from_numpy(np.empty(0, dtype)).dtype
        np.testing.assert_array_equal(t.cpu().numpy(), w)
