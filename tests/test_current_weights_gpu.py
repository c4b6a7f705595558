"""Every evaluation computes with the parameters as they are when it starts, however they were changed: the bf16 copies that the
Linear layers compute with may not be older.  Version counters do not see a graph's replay, writes through ``.data`` or
writes to a flat buffer that the parameters are views of."""
import io
import threading

import pytest
import torch

from matterformer_b200.dp import GraphedTrainStep, build_edm_net
from matterformer_b200.linear import linear_bf16
from matterformer_b200.sampler import GraphedDenoiser, build_pad_mask, edm_sample
from matterformer_b200.synthetic import config5_batch
from matterformer_b200.trunk import EDMLoss

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
COUNTS = [9, 6, 4, 1]


def _net(seed=0):
    net = build_edm_net(d_model=128, n_heads=2, n_layers=2, seed=seed).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    with torch.no_grad():
        for p in net.parameters():  # (the modulation and the pair head start at zero)
            p.add_(torch.randn(p.shape, device=DEV, generator=g) * 0.05)
    return net


def _twin(net):
    """A network that has computed nothing yet, with the parameters that ``net`` has now."""
    twin = build_edm_net(d_model=128, n_heads=2, n_layers=2, seed=7).to(DEV)
    twin.load_state_dict(net.state_dict())
    return twin


def _denoiser(net, n):
    pad = build_pad_mask(n)
    with torch.no_grad():
        return GraphedDenoiser(net, torch.zeros(*pad.shape, 6, device=DEV), torch.zeros(*pad.shape, 3, device=DEV), pad, None,
                               torch.bfloat16)  # fmt: skip


def _sample(net, n, denoiser=None, graph=None):
    torch.manual_seed(3)
    a, c, _ = edm_sample(net, n, num_steps=3, autocast_dtype=torch.bfloat16, denoiser=denoiser, use_cuda_graph=graph)
    return torch.cat([a, c], -1)


def _net_and_change(route):
    """A network, and a function that changes all its parameters by the given route: their version counters do not notice."""
    net = _net()
    params = list(net.parameters())
    if route == "data":

        def change():
            for p in params:
                p.data.mul_(1.5)

    elif route == "flat":
        width = [-(-p.numel() // 128) * 128 for p in params]
        flat, at = torch.zeros(sum(width), device=DEV), 0
        for p, w in zip(params, width):
            view = flat[at : at + p.numel()].view(p.shape)
            view.copy_(p.data)
            p.data, at = view, at + w

        def change():
            flat.mul_(1.5)

    else:
        opt = torch.optim.AdamW(params, lr=3e-3, fused=True, capturable=True)
        batch = {k: v.to(DEV) for k, v in config5_batch(8, seed=1).items() if k != "num_atoms"}
        step = GraphedTrainStep(net, EDMLoss(sigma_data=1.0), opt, batch, warmup=3)
        step()

        def change(keep=opt):  # (the captured step reads and writes the optimizer's state)
            step()

    return net, change


@pytest.mark.parametrize("route", ["data", "flat", "replay"])
@pytest.mark.parametrize("kept", [True, False])
def test_samples_come_from_the_current_weights(route, kept):
    (net, change), n = _net_and_change(route), torch.tensor(COUNTS, device=DEV)
    denoiser = _denoiser(net, n) if kept else None
    before = _sample(net, n, denoiser)
    change()
    after = _sample(net, n, denoiser)
    expect = _sample(_twin(net), n)
    assert (expect - before).abs().max() > 1e-2  # the change shows
    torch.testing.assert_close(after, expect, atol=1e-5, rtol=1e-5)  # the same kernels on the same weights


def test_one_evaluation_of_a_kept_denoiser_follows_too():
    (net, change), n = _net_and_change("data"), torch.tensor(COUNTS, device=DEV)
    denoiser = _denoiser(net, n)
    g = torch.Generator(device=DEV).manual_seed(0)
    pad = build_pad_mask(n)
    a, c = (torch.randn(*pad.shape, k, device=DEV, generator=g) * ~pad[..., None] for k in (6, 3))
    first = [t.clone() for t in denoiser(a, c, 0.7)]
    change()
    second = [t.clone() for t in denoiser(a, c, 0.7)]
    expect = _denoiser(_twin(net), n)(a, c, 0.7)
    assert (first[0] - second[0]).abs().max() > 1e-2
    for x, y in zip(second, expect):
        torch.testing.assert_close(x, y, atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("route", ["data", "flat", "replay"])
@pytest.mark.parametrize("grad", [False, True])
def test_eager_passes_compute_with_the_current_weights(route, grad):
    net, change = _net_and_change(route)
    g = torch.Generator(device=DEV).manual_seed(0)
    pad = build_pad_mask(torch.tensor(COUNTS, device=DEV))
    a, c = (torch.randn(*pad.shape, k, device=DEV, generator=g) * ~pad[..., None] for k in (6, 3))
    sigma = torch.ones(len(COUNTS), device=DEV)

    def run(m):
        with torch.set_grad_enabled(grad), torch.autocast("cuda", dtype=torch.bfloat16):
            out = m(a, c, pad, sigma)
        grads = torch.autograd.grad(sum(t.float().square().sum() for t in out), list(m.parameters())) if grad else []
        return [*out, *grads]

    before = run(net)
    change()
    after, expect = run(net), run(_twin(net))
    assert (expect[0] - before[0]).abs().max() > 1e-2
    for x, y in zip(after, expect):
        torch.testing.assert_close(x, y, atol=1e-5 * max(1.0, y.abs().max().item()), rtol=1e-5)


def test_single_layers_compute_with_the_current_weights():
    lin = torch.nn.Linear(64, 32).to(DEV)
    x = torch.randn(4, 64, device=DEV).bfloat16()
    with torch.no_grad():
        linear_bf16(x, lin.weight, lin.bias)
        lin.weight.data.mul_(2.0)
        y = linear_bf16(x, lin.weight, lin.bias)
        assert torch.equal(y, torch.nn.functional.linear(x, lin.weight.bfloat16(), lin.bias.bfloat16()))


def test_a_pass_between_forward_and_backward_leaves_the_gradient_alone():
    """Sampling (or a second micro-batch) between a forward pass and its backward pass is ordinary use."""
    net, n = _net(), torch.tensor(COUNTS, device=DEV)
    pad = build_pad_mask(n)
    g = torch.Generator(device=DEV).manual_seed(0)
    a, c = (torch.randn(*pad.shape, k, device=DEV, generator=g) * ~pad[..., None] for k in (6, 3))
    sigma = torch.ones(len(COUNTS), device=DEV)
    grads = []
    for between in (False, True):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out = net(a, c, pad, sigma)
        if between:
            _sample(net, n, graph=False)
        grads.append(torch.autograd.grad(sum(t.float().square().sum() for t in out), list(net.parameters())))
    for x, y in zip(*grads):
        assert torch.equal(x, y)


def test_copies_are_no_part_of_the_module():
    """Saved and copied networks are as large after a pass as before it."""

    def size(net):
        f = io.BytesIO()
        torch.save(net, f)
        return f.tell()

    net, n = _net(), torch.tensor(COUNTS, device=DEV)
    before = size(net)
    _sample(net, n, graph=False)
    assert size(net) <= before + 4096
    assert not any(vars(p) for p in net.parameters())


def test_copies_belong_to_one_thread():
    from matterformer_b200.linear import KeptBf16Copies, bf16_copies, bf16_copy

    p = torch.nn.Parameter(torch.randn(16, 128, device=DEV))
    seen = {}

    def other():
        seen["copy"] = bf16_copy(p)
        with bf16_copies([p]):
            seen["own"] = bf16_copy(p)

    kept = KeptBf16Copies()
    with kept.in_use(), bf16_copies([p]) as stacked:
        mine = bf16_copy(p)
        assert stacked == [] and bf16_copy(p) is mine
        t = threading.Thread(target=other)
        t.start()
        t.join()
    assert len({t.data_ptr() for t in (mine, seen["copy"], seen["own"])}) == 3
    p.data.add_(1.0)
    assert not torch.equal(mine, p.detach().bfloat16())
    kept.refresh()
    assert torch.equal(mine, p.detach().bfloat16())
    assert torch.equal(bf16_copy(p), p.detach().bfloat16())


def test_stacked_copies_and_odd_sizes():
    """Copies of parameters whose sizes are no multiple of the buffer's alignment, next to stacks."""
    from matterformer_b200.linear import bf16_copies, bf16_copy

    g = torch.Generator(device=DEV).manual_seed(0)
    new = lambda *s: torch.nn.Parameter(torch.randn(*s, device=DEV, generator=g))  # noqa: E731
    params, stacks = [new(6), new(3, 128), new(1, 7), new(256), None], [[new(48, 8), new(48, 8)], [new(48), new(48), new(48)]]
    with bf16_copies(params + stacks[0], stacks) as made:
        for p in [*params[:-1], *stacks[0], *stacks[1]]:
            assert torch.equal(bf16_copy(p), p.detach().bfloat16())
            assert bf16_copy(p).data_ptr() % 16 == 0
        for m, stack in zip(made, stacks):
            assert m.data_ptr() % 256 == 0 and torch.equal(m, torch.cat([p.detach().bfloat16() for p in stack]))


@pytest.mark.parametrize("how", ["data", "assign", "layer"])
def test_a_kept_denoiser_follows_parameters_that_move(how):
    """Parameters placed in new memory (a swap of ``.data``, a loaded checkpoint that is assigned, a replaced layer): the captured
    evaluation reads some of them in place and has to be captured anew."""
    net, n = _net(), torch.tensor(COUNTS, device=DEV)
    denoiser = _denoiser(net, n)
    before = _sample(net, n, denoiser)
    if how == "data":
        for p in net.parameters():
            p.data = p.data * 1.5
    elif how == "assign":
        net.load_state_dict({k: v * 1.5 for k, v in net.state_dict().items()}, assign=True)
    else:
        old = net.model.pair_head[2]
        net.model.pair_head[2] = torch.nn.Linear(old.in_features, 1).to(DEV)
        net.model.atom_head[3] = torch.nn.Linear(128, 6).to(DEV)
    filler = [torch.full((1 << 20,), float("nan"), device=DEV) for _ in range(4)]  # what was freed is written over
    after = _sample(net, n, denoiser)
    expect = _sample(_twin(net), n)
    del filler
    assert (expect - before).abs().max() > 1e-2
    torch.testing.assert_close(after, expect, atol=1e-5, rtol=1e-5)


def test_a_capture_inside_an_autocast_region_takes_no_casts_from_it():
    """Above 32 tokens the MHA layers are torch's, whose weights autocast casts and keeps until its outermost region ends: casts
    made before the capture would stay in the graph."""
    net, n = _net(), torch.tensor([40, 33], device=DEV)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        denoiser = _denoiser(net, n)
        before = _sample(net, n, denoiser)
        for p in net.parameters():
            p.data.mul_(1.5)
        after, expect = _sample(net, n, denoiser), _sample(_twin(net), n)
    assert (expect - before).abs().max() > 1e-2
    torch.testing.assert_close(after, expect, atol=1e-5, rtol=1e-5)
