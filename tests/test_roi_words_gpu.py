"""CONTOUR ROIs by table: the device's mapping of every voxel against the search over the runs written
out in Python, for runs in order (the table holds them) and for arrays no table can hold (out of
order, overlapping, accumulated lengths that are not theirs: the search stays), on grids about whole
words of 32 voxels."""
import numpy as np
import pytest

from moquimc_gb300 import capi

pytestmark = pytest.mark.gpu


def _search(start, stride, acc, v):
    first, count = 0, len(start)
    while count > 0:
        step = count // 2
        if start[first + step] <= v:
            first, count = first + step + 1, count - step - 1
        else:
            count = step
    c = first - 1
    if c < 0:
        return -1, -1
    d = (int(v) - int(start[c])) & 0xFFFFFFFF
    if d >= stride[c]:
        return -1, -1
    return 1, d + (int(acc[c - 1]) if c > 0 else 0)


def _runs(kind, n, rng):
    m = rng.random(n) < 0.4
    m[rng.integers(n)] = True
    edge = np.flatnonzero(np.diff(np.concatenate([[0], m.view(np.int8), [0]])))
    start, stride = edge[0::2].astype(np.uint32), (edge[1::2] - edge[0::2]).astype(np.uint32)
    if kind == "touching":                       # every run cut in two that touch
        cut = np.maximum(stride // 2, 1)
        start = np.stack([start, start + cut], 1).ravel().astype(np.uint32)
        stride = np.stack([cut, stride - cut], 1).ravel().astype(np.uint32)
    if kind == "unsorted":
        p = rng.permutation(len(start))
        start, stride = start[p], stride[p]
    if kind == "overlapping":
        stride = (stride + 3).astype(np.uint32)
    acc = np.cumsum(stride).astype(np.uint32)
    if kind == "accumulated":
        acc = (acc + np.arange(len(acc)) % 3).astype(np.uint32)
    return start, stride, acc


@pytest.mark.parametrize("kind", ["ordered", "touching", "unsorted", "overlapping", "accumulated"])
@pytest.mark.parametrize("nxyz", [(1, 1, 1), (31, 1, 1), (8, 2, 2), (11, 3, 1), (17, 13, 9)])
@pytest.mark.parametrize("stat", [False, True])
def test_contour_mapping(gpu_ctx_factory, kind, nxyz, stat):
    n = int(np.prod(nxyz))
    start, stride, acc = _runs(kind, n, np.random.default_rng(n))
    c = gpu_ctx_factory()
    cid = c.add_child(*[np.arange(k + 1, dtype=np.float32) for k in nxyz])
    if stat:
        sid = c.add_stat_scorers(cid, capi.ROI_CONTOUR, start, stride, acc)[0]
    else:
        sid = c.add_scorer(cid, capi.DOSE_W, capi.ROI_CONTOUR, start, stride, acc)
    idx, mask = c.eval_roi(sid, np.arange(n))
    want = np.array([_search(start, stride, acc, v) for v in range(n)])
    np.testing.assert_array_equal(idx, want[:, 0])
    np.testing.assert_array_equal(mask, want[:, 1])
