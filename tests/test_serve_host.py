"""The server's estimate of a request's device memory (no GPU needed)."""
import numpy as np

from chidg_b200 import mesh, serve


def _blocks_and_vectors(pat, nkrylov):
    nr, nc = (np.asarray(d, dtype=np.int64) for d in pat.block_dims())
    low = np.asarray(pat.blk_col_elem) <= np.asarray(pat.blk_row_elem)
    return 8 * int((nr * nc).sum() + (nr * nc)[low].sum()) + 8 * pat.vector_size() * (2 * (nkrylov + 1) + 6)


def test_request_bytes_counts_the_sweeps_scratch():
    """Backward partial sums of an interior row of 135 equations: three slices of
    its three upper entries and of inv(D); the task lists come on top."""
    pat = mesh.box_pattern(24, 24, 24, 5, 27)
    interior = 23 ** 3
    extra = serve.request_bytes(pat, 30) - _blocks_and_vectors(pat, 30)
    scratch = 8 * 135 * 3 * 4 * interior
    assert scratch <= extra < 1.5 * scratch


def test_request_bytes_of_one_task_rows():
    """Rows of up to 64 equations: a vector an entry, and a task in each list."""
    pat = mesh.box_pattern(3, 1, 1, 5, 8)
    extra = serve.request_bytes(pat, 30) - _blocks_and_vectors(pat, 30)
    assert 8 * 40 * 3 <= extra <= 8 * 40 * 3 + 3 * 4 * 128
