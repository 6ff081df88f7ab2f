"""What the C++ autograd nodes compute for each way of asking: only the gradients that the running
backward needs, with the values of a full backward."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture()
def setup():
    from permutohedral_encoding_b200 import PermutoEncoding
    torch.manual_seed(11)
    m = PermutoEncoding(3, 2 ** 12, 6, 2, np.geomspace(1.0, 1e-2, 6))
    with torch.no_grad():
        m.lattice_values.uniform_(-1, 1)
    pos = torch.rand(500, 3, device=DEV, requires_grad=True)
    return m, pos, torch.randn(500, 12, device=DEV)


def _close(a, b):
    assert torch.all((a - b).abs() <= 1e-4 * b.abs().amax())


def test_restricted_backwards_match_the_full_one(setup):
    m, pos, go = setup
    m(pos).backward(go)
    want_v, want_p = m.lattice_values.grad.clone(), pos.grad.clone()
    m.lattice_values.grad = pos.grad = None
    (p,) = torch.autograd.grad(m(pos), pos, go)
    _close(p, want_p)
    (v,) = torch.autograd.grad(m(pos), m.lattice_values, go)
    _close(v, want_v)
    torch.autograd.backward([m(pos)], [go], inputs=[m.lattice_values])
    _close(m.lattice_values.grad, want_v)
    assert pos.grad is None


def test_double_backward_and_hooks(setup):
    """create_graph keeps the position gradient differentiable; hooks installed between forward and
    backward are called, with the gradients they return used."""
    m, pos, go = setup
    go.requires_grad_(True)
    dpg = torch.randn(500, 3, device=DEV)
    (p,) = torch.autograd.grad(m(pos), pos, go, create_graph=True)
    p.backward(dpg)
    want_v, want_g = m.lattice_values.grad.clone(), go.grad.clone()
    assert torch.count_nonzero(want_g) > 0
    m.lattice_values.grad = go.grad = None
    (p,) = torch.autograd.grad(m(pos), pos, go, create_graph=True)
    m.lattice.double_backward_hook = lambda g: 2.0 * g
    p.backward(dpg)
    m.lattice.double_backward_hook = None
    _close(m.lattice_values.grad, 2.0 * want_v)
    _close(go.grad, want_g)

    pos2 = pos.detach()
    m.lattice_values.grad = None
    m(pos2).backward(go.detach())
    want = m.lattice_values.grad.clone()
    m.lattice_values.grad = None
    out = m(pos2)
    seen = []

    def hook(lattice, inp, grad):
        seen.append(grad.shape)
        g, p = lattice.backward(inp, grad)
        return 3.0 * g, p

    m.lattice.backward_hook = hook
    out.backward(go.detach())
    m.lattice.backward_hook = None
    assert seen == [go.shape]
    _close(m.lattice_values.grad, 3.0 * want)


def test_saved_tensors_are_guarded(setup):
    m, pos, go = setup
    out = m(pos)
    with torch.no_grad():
        m.lattice_values.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(go)


@pytest.mark.parametrize("n", [33, 2 ** 19 + 77])
@pytest.mark.parametrize("d,feat,levels", [(2, 2, 3), (3, 2, 9), (3, 4, 5), (4, 8, 3), (6, 2, 5), (7, 4, 2)])
def test_both_orders_in_one_backward(d, feat, levels, n):
    """A loss on the features and on the position gradient: the table gradient of one backward is the
    sum of the two separate ones (1e-4 * sum|addend|, as for any order of the fp32 sums), whichever
    node runs first, restricted or not, and again when the graph is kept."""
    from permutohedral_encoding_b200 import PermutoEncoding
    torch.manual_seed(d)
    m = PermutoEncoding(d, 2 ** 10, levels, feat, np.geomspace(1.0, 1e-2, levels))
    with torch.no_grad():
        m.lattice_values.uniform_(-1, 1)
    pos = torch.rand(n, d, device=DEV, requires_grad=True)
    go = torch.randn(n, m.output_dims(), device=DEV)
    up = torch.randn(n, m.output_dims(), device=DEV, requires_grad=True)
    dpg = torch.randn(n, d, device=DEV)

    def graph():
        out = m(pos)
        (normal,) = torch.autograd.grad(out, pos, up, create_graph=True)
        return out, normal

    out, normal = graph()
    first = torch.autograd.grad(out, m.lattice_values, go, retain_graph=True)[0]
    second, want_up = torch.autograd.grad(normal, [m.lattice_values, up], dpg)
    want = first + second
    bound = 1e-4 * (first.abs() + second.abs()) + 1e-5 * want.abs().amax()

    def check(got, got_up):
        assert torch.all((got - want).abs() <= bound)
        assert torch.all((got_up - want_up).abs() <= 1e-5 * want_up.abs().amax())

    check(*torch.autograd.grad(graph(), [m.lattice_values, up], [go, dpg]))
    out, normal = graph()
    for _ in range(2):
        m.lattice_values.grad = up.grad = None
        torch.autograd.backward([out, normal], [go, dpg], inputs=[m.lattice_values, up], retain_graph=True)
        check(m.lattice_values.grad, up.grad)
    m.lattice_values.grad = up.grad = pos.grad = None
    torch.autograd.backward([normal, out], [dpg, go])          # everything, the position gradient of `out` too
    check(m.lattice_values.grad, up.grad)
    assert pos.grad is not None
    # the features' part runs first when the other part hangs on it
    out, normal = graph()
    m.lattice_values.grad = up.grad = None
    (normal * dpg).sum().backward()
    out2, _ = graph()
    check(m.lattice_values.grad + torch.autograd.grad(out2, m.lattice_values, go)[0], up.grad)


def _large(n=2 ** 18 + 5, levels=16):
    from permutohedral_encoding_b200 import PermutoEncoding
    torch.manual_seed(3)
    m = PermutoEncoding(3, 2 ** 10, levels, 2, np.geomspace(1.0, 1e-2, levels))
    with torch.no_grad():
        m.lattice_values.uniform_(-1, 1)
    return m, torch.rand(n, 3, device=DEV, requires_grad=True), torch.randn(n, 2 * levels, device=DEV)


def test_a_backward_frees_what_the_graph_kept():
    """The engine frees the saved tensors, the spatial order among them, with a backward that does not keep
    the graph, even while its output lives; the pose case runs both nodes of a create_graph backward."""
    m, pos, go = _large()
    out = m(pos)
    held = torch.cuda.memory_allocated()
    out.backward(go, inputs=[m.lattice_values])
    m.lattice_values.grad = None
    assert held - torch.cuda.memory_allocated() >= 16 * pos.shape[0]
    with pytest.raises(RuntimeError, match="second time"):
        out.backward(go)
    before = torch.cuda.memory_allocated()
    out2 = m(pos)
    (normal,) = torch.autograd.grad(out2, pos, go, create_graph=True)
    torch.autograd.backward([out2, normal], [go, torch.ones_like(normal)], inputs=[m.lattice_values])
    kept = sum(t.numel() * 4 for t in (out2, normal, m.lattice_values.grad))
    assert torch.cuda.memory_allocated() - before <= kept + 4096


@pytest.mark.parametrize("large", [False, True])
def test_saved_tensor_hooks_see_and_replace_what_a_node_keeps(setup, large):
    m, pos, go = _large() if large else setup
    window = None if large else torch.rand(m.nr_levels, device=DEV)   # with a window on the device nothing is ordered

    def grads(out):
        return torch.autograd.grad(out, [m.lattice_values, pos], go)

    want_v, want_p = grads(m(pos, window))
    seen = []

    def keep(t):
        seen.append(t)
        return t

    def same(ts):
        return sorted((tuple(t.shape), t.dtype) for t in ts)

    with torch.autograd.graph.saved_tensors_hooks(keep, lambda t: t):
        out = m(pos, window)
    assert same(seen) == same([m.lattice_values, pos, m.anneal_window if large else window])
    got_v, got_p = grads(out)
    _close(got_v, want_v)
    _close(got_p, want_p)
    # the table gradient is linear in the window, the position gradient in window and values
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t * 2 if t.shape != pos.shape else t):
        out = m(pos, window)
    got_v, got_p = grads(out)
    _close(got_v, 2 * want_v)
    _close(got_p, 4 * want_p)
    # moved points, first order and second order
    where = (pos.detach() + 0.25).requires_grad_(True)
    (want_n,) = torch.autograd.grad(m(where, window), where, go, create_graph=True)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t + 0.25 if t.shape == pos.shape else t):
        (normal,) = torch.autograd.grad(m(pos, window), pos, go, create_graph=False)
        _close(normal, want_n.detach())
    with torch.autograd.graph.save_on_cpu():
        (normal,) = torch.autograd.grad(m(where, window), where, go.requires_grad_(True), create_graph=True)
        got = torch.autograd.grad(normal.sum(), [m.lattice_values, go])
    want = torch.autograd.grad(torch.autograd.grad(m(where, window), where, go, create_graph=True)[0].sum(), [m.lattice_values, go])
    for a, b in zip(got, want):
        _close(a, b)


def test_checkpointed_batches_match():
    from torch.utils.checkpoint import checkpoint
    m, pos, go = _large()
    want = torch.autograd.grad(m(pos), [m.lattice_values, pos], go)
    got = torch.autograd.grad(checkpoint(m, pos, use_reentrant=False), [m.lattice_values, pos], go)
    for a, b in zip(got, want):
        _close(a, b)


@pytest.mark.parametrize("d,feat,levels", [(2, 2, 13), (3, 4, 12), (4, 8, 8), (6, 2, 16), (7, 8, 8)])
def test_both_orders_in_one_backward_of_an_ordered_batch(d, feat, levels):
    """The same on batches that the module puts into spatial order."""
    from permutohedral_encoding_b200 import _native as nat
    n = 2 ** 19 + 77
    assert nat.lib.permuto_order_pays(nat.PermutoConfig(d, feat, levels, 2 ** 10, 0, 1.0, 0, 0), n, nat.ORDER_POSITIONS)
    test_both_orders_in_one_backward(d, feat, levels, n)
