"""The differentiated iterations wait for torch's streams on the device, not on the host: results and gradients
with inputs made and dropped on other torch streams, two models queued in turn, memory reused at once, against
the same calls made one at a time. The adjoint's sums are atomic, so their order differs: 1e-12 of the largest."""
import pytest

from atjup_b200.params import LIN_FIELDS
from test_iteration_adjoint import prepared

torch = pytest.importorskip("torch")


def gradients(m, x, seed):
    from atjup_b200.autograd import iterations
    out = iterations(m, x, 2, start=2)
    g = torch.autograd.grad(out, x, grad_outputs=seed)
    return [y.detach() for y in out], g


@pytest.mark.gpu
def test_streams_and_reused_memory():
    models = [prepared((9, 13, 25), s) for s in (1, 2)]
    models = [m for _, _, m in models]
    km = models[0].shape[2]
    want, state, seeds = [], [], []
    for q, m in enumerate(models):
        x = [t.clone() for t in m.state_tensors(LIN_FIELDS)]
        gen = torch.Generator(device="cuda").manual_seed(q)
        seed = [torch.randn(t.shape, dtype=t.dtype, device="cuda", generator=gen) for t in x]
        want.append(gradients(m, [t.clone().requires_grad_() for t in x], seed))
        torch.cuda.synchronize()
        state.append(x)
        seeds.append(seed)
    streams = [torch.cuda.Stream() for _ in models]
    other = torch.cuda.Stream()
    for _ in range(5):
        got = []
        for m, x, seed, s in zip(models, state, seeds, streams):
            with torch.cuda.stream(other):
                y = [t.clone().requires_grad_() for t in x]
                sd = [t.clone() for t in seed]
            s.wait_stream(other)
            with torch.cuda.stream(s):
                got.append(gradients(m, y, sd))
            del y, sd
            with torch.cuda.stream(other):      # takes the dropped tensors' memory
                junk = [torch.full_like(t, float("nan")) for t in x + seed]
            del junk
        torch.cuda.synchronize()
        for (o, g), (wo, wg) in zip(got, want):
            for a, b in zip([*o, *g], [*wo, *wg]):
                assert (a - b)[:, :, :km].abs().max() <= 1e-12 * b[:, :, :km].abs().max()
    for m in models:
        m.close()
