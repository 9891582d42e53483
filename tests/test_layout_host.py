"""Packed layouts of empty batches and empty problems (no GPU)."""
import torch

from pot_gb300.batch import RaggedLayout


def test_empty_batch():
    lay = RaggedLayout([], [], torch.float32, torch.device("cpu"))
    assert lay.B == 0 and lay.total_m == lay.total_r == lay.total_c == 0


def test_empty_problems_stay_off_the_one_read_kernel():
    """Its row shares and bulk copies want a row and a column of every problem."""
    for rows, cols in (([0, 3], [4, 4]), ([3, 3], [4, 0])):
        assert RaggedLayout(rows, cols, torch.float32, torch.device("cpu")).max_ldm == 0
    assert RaggedLayout([2, 3], [4, 7], torch.float32, torch.device("cpu")).max_ldm == 8
