"""The Adam update of a list of tensors (sizes around a CTA's 1,024 values, more tensors
than a launch takes, empty ones) and the flipped weights (channel counts around the
32 x 32 tiles)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from hemelb_gb300 import nn  # noqa: E402
from oracle import nn_oracle as O  # noqa: E402


@pytest.mark.parametrize("sizes", [(1,), (1023, 1024, 1025), (0, 5, 0, 4096, 7, 0), tuple(range(1, 71)), (200_003, 3)])
def test_adam_list_matches_the_oracle_tensor_by_tensor(sizes):
    rng = np.random.default_rng(len(sizes))
    w = [rng.standard_normal(n) for n in sizes]
    g = [rng.standard_normal(n) for n in sizes]
    tw = [torch.tensor(a, dtype=torch.float32, device="cuda") for a in w]
    tg = [torch.tensor(a, dtype=torch.float32, device="cuda") for a in g]
    tm, tv = [torch.zeros_like(a) for a in tw], [torch.zeros_like(a) for a in tw]
    tb = [a.to(torch.bfloat16) if i % 2 == 0 else None for i, a in enumerate(tw)]
    ref = [(a.double().cpu().numpy(), np.zeros(a.numel()), np.zeros(a.numel())) for a in tw]
    for step in (1, 2, 3):
        nn.adam_list(list(zip(tw, tb, tg, tm, tv)), 1e-2, step)
        ref = [O.adam_step(r[0], a.double().cpu().numpy(), r[1], r[2], 1e-2, step) for r, a in zip(ref, tg)]
    for a, b, (r, _, _) in zip(tw, tb, ref):
        # three updates of at most 1e-2 with some ten FP32 roundings each, and three of w
        bound = 3 * (10 * 1e-2 + np.abs(r) + 1e-2) * 2.0 ** -23
        assert (np.abs(a.double().cpu().numpy() - r) <= bound).all()
        if b is not None:
            assert torch.equal(b, a.to(torch.bfloat16))


def test_adam_list_refuses_tensors_of_other_sizes():
    a = [torch.zeros(n, device="cuda") for n in (4, 4, 3, 4)]
    with pytest.raises(ValueError):
        nn.adam_list([(a[0], None, a[1], a[2], a[3])], 1e-3, 1)


@pytest.mark.parametrize("shape", [(1, 16, 16), (27, 48, 80), (3, 33, 7), (27, 1, 65), (2, 32, 31), (1, 300, 16)])
def test_flipped_weights(shape):
    w = torch.arange(int(np.prod(shape)), device="cuda").remainder(251).to(torch.bfloat16).view(shape)
    wt = torch.empty((shape[0], shape[2], shape[1]), dtype=torch.bfloat16, device="cuda")
    nn.flip_transpose(w, wt)
    assert torch.equal(wt, w.flip(0).transpose(1, 2))
