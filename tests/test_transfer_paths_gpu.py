"""State transfers from and to page-locked, pageable and mixed host arrays, at
sizes on both sides of the limit of the direct path: every element arrives,
bit for bit, and arrays that are left out stay as they were."""
import numpy as np
import pytest

from ixchel2d_b200 import Simple2D, cases

pytestmark = pytest.mark.gpu
KEYS = ("u", "v", "p", "T", "u_ant", "v_ant", "T_ant")


def _array(shape, pinned, keep):
    import torch
    n = int(np.prod(shape))
    if not pinned:
        return np.empty(shape, order="F")
    t = torch.empty(n + 3, dtype=torch.float64).pin_memory()
    keep.append(t)
    return t.numpy()[3:].reshape(shape, order="F")  # not at the start of its allocation


@pytest.mark.parametrize("kind", ["pinned", "pageable", "mixed", "some"])
@pytest.mark.parametrize("mi, nj", [(4, 4), (33, 18), (257, 130), (701, 426), (700, 428)])
def test_round_trip(has_gpu, mi, nj, kind):
    if not has_gpu:
        pytest.skip("no CUDA device")
    case, keep = cases.lid_driven_mixed(mi, nj), []
    shapes = cases.shapes(mi, nj)
    rng = np.random.default_rng(mi + nj)
    keys = KEYS if kind != "some" else ("v", "T", "T_ant")
    up = {k: _array(shapes[k], kind != "pageable" and not (kind == "mixed" and k == "p"), keep) for k in keys}
    down = {k: _array(shapes[k], kind != "pageable" and not (kind == "mixed" and k == "T"), keep) for k in KEYS}
    for a in up.values():
        a[...] = rng.uniform(-1, 1, a.shape)
    with Simple2D.from_case(case) as s:
        before = s.download()
        s.upload(up)
        s.download(down)
        again = s.download()
    for k in KEYS:
        want = up[k] if k in up else before[k]
        assert np.array_equal(down[k], want) and np.array_equal(again[k], want), k
