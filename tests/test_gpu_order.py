"""Spatial order of a batch: it is a permutation that carries the coordinates, and every operation
gives with it what it gives without it -- forward and per-point gradients bit for bit (a point's
arithmetic does not depend on its neighbours), table gradients within the bound of summing the same
fp32 addends in another order, 1e-4 * sum|addend|.  Sizes around the kernels' edges: one point, one
thread's group of points, warps, blocks, several blocks; feature rows with and without 32-byte
alignment; identical points and points far outside the bulk of the batch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def nat():
    from permutohedral_encoding_b200 import _native
    return _native


def _setup(nat, d, feat, levels, n, seed, concat=False, half=False, shape="box"):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    cap = 2 ** 12 if d != 4 else 3001
    shift = torch.randn((levels, d), device=DEV, generator=gen) * 10
    fx = nat.EncodingFixedParams(d, cap, levels, feat, np.geomspace(1.0, 1e-3, levels), shift, concat, 0.5)
    enc = nat.EncodingWrapper.create(d, feat, fx)
    table = torch.randn((levels, cap, feat), device=DEV, generator=gen)
    pos = torch.rand((n, d), device=DEV, generator=gen) * 2 - 1
    if shape == "same":
        pos[:] = pos[0].clone()
    elif shape == "outliers":
        pos[::97] *= 1e6
        pos[1::101, 0] = float("inf")
    elif shape == "flat":
        pos[:, 1:] = 0.25
    window = torch.rand(levels, device=DEV, generator=gen)
    window[0] = 0.0
    inp = nat.EncodingInput(table.half() if half else table, pos, window, True, True)
    go = torch.randn((n, enc.output_width()), device=DEV, generator=gen)
    return enc, inp, go, torch.randn((n, d), device=DEV, generator=gen)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 255, 257, 1025, 30011])
@pytest.mark.parametrize("d,feat,levels,concat,half", [(2, 2, 7, False, False), (3, 2, 8, False, True), (3, 2, 5, True, False),
                                                       (4, 4, 5, False, False), (6, 2, 12, False, False), (3, 8, 3, True, True),
                                                       (7, 4, 34, False, False)])
def test_ordered_equals_unordered(nat, n, d, feat, levels, concat, half):
    enc, inp, go, dpg = _setup(nat, d, feat, levels, n, n + d, concat, half)
    only_table = nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, True, False)
    only_pos = nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, False, True)

    def run(order):
        inp.m_order = only_table.m_order = only_pos.m_order = order
        tables = [enc.backward(only_table, go)[0], enc.backward(inp, go)[0], enc.double_backward_from_positions(inp, dpg, go)[0]]
        rows = [enc.forward(inp), enc.double_backward_from_positions(inp, dpg, go)[1]]
        points = [enc.backward(inp, go)[1], enc.backward(only_pos, go)[1]]
        return tables, rows, points

    plain, ordered = run(None), run(enc.order(inp))
    magnitude = [enc.backward(only_table, go.abs())[0]] * 2 + [plain[0][2].abs().amax().expand_as(plain[0][2])]
    for a, b, m in zip(plain[0], ordered[0], magnitude):
        assert torch.all((a - b).abs() <= 1e-4 * m + 1e-6 * m.amax())
    for a, b in zip(plain[1], ordered[1]):
        assert torch.equal(a, b)
    for a, b in zip(plain[2], ordered[2]):   # sums over sweeps of levels: same addends, another grouping
        assert torch.all((a - b).abs() <= 1e-5 * a.abs().amax())


@pytest.mark.parametrize("shape", ["box", "same", "outliers", "flat"])
@pytest.mark.parametrize("d,n", [(2, 5000), (3, 1), (3, 4097), (5, 9000), (3, 2 ** 22 + 1025)])
def test_order_is_a_permutation_with_coordinates(nat, shape, d, n):
    enc, inp, _, _ = _setup(nat, d, 2, 4, n, 3, shape=shape)
    words = 4 if d <= 3 else 8
    rec = enc.order(inp)[:4 * words * n].view(torch.int32).view(n, words)
    idx = rec[:, words - 1].long()
    assert torch.equal(torch.sort(idx).values, torch.arange(n, device=DEV))
    assert torch.equal(rec[:, :d].contiguous(), inp.m_positions_raw[idx].view(torch.int32))


def test_module_orders_large_batches(nat):
    """The module's own rule: above the threshold the batch is ordered, and nothing shows but time."""
    from permutohedral_encoding_b200 import PermutoEncoding
    torch.manual_seed(5)
    m = PermutoEncoding(3, 2 ** 14, 8, 2, np.geomspace(1.0, 1e-3, 8))
    pos = torch.rand(2 ** 19 + 77, 3, device=DEV)
    inp = nat.EncodingInput(m.lattice_values.detach(), pos, m.anneal_window, False, False)
    assert m.lattice.order(inp, nat.ORDER_TRAINING) is not None
    with torch.no_grad():
        assert torch.equal(m(pos), m.lattice.forward(inp))
    small = nat.EncodingInput(m.lattice_values.detach(), pos[:1000], m.anneal_window, False, False)
    assert m.lattice.order(small, nat.ORDER_TRAINING) is None


def test_large_batches_sum_as_without_an_order(nat):
    """Beyond 2^22 points the table gradients -- first order, second order, and a loss with both -- are fp32
    sums in the sequence of the batch: per level they differ from the unordered kernels' by no more than those
    differ from themselves in another run.  The bound is 1.3 times: a level's deviation is a 2-norm over a
    thousand slots or more, which varies by a few per cent (0.97-1.12 measured); sums in spatial order are
    at 1.6-2.3."""
    from permutohedral_encoding_b200 import PermutoEncoding
    n, levels = 2 ** 22 + 2051, 12
    torch.manual_seed(21)
    m = PermutoEncoding(3, 2 ** 15, levels, 2, np.geomspace(0.035, 1e-3, levels))
    with torch.no_grad():
        m.lattice_values.uniform_(-1, 1)
    pos = (torch.rand(n, 3, device=DEV) - 0.5).requires_grad_(True)
    go, dpg = torch.randn(n, 2 * levels, device=DEV), torch.randn(n, 3, device=DEV)
    inp = nat.EncodingInput(m.lattice_values.detach(), pos.detach(), m.anneal_window, True, False)
    assert m.lattice.order(inp, nat.ORDER_POSITIONS) is not None

    def first():
        return m.lattice.backward(inp, go)[0]

    def second():
        return m.lattice.double_backward_from_positions(inp, dpg, go)[0]

    def grads(*, features, normals):
        m.lattice_values.grad = None
        out = m(pos)
        heads = [(out, go)] if features else []
        if normals:
            heads.append((torch.autograd.grad(out, pos, go, create_graph=True)[0], dpg))
        torch.autograd.backward([h for h, _ in heads], [g for _, g in heads], inputs=[m.lattice_values])
        return m.lattice_values.grad

    def off(a, b):
        return (a.double() - b.double()).flatten(1).norm(dim=1)

    for plain, got in ((first, grads(features=True, normals=False)), (second, grads(features=False, normals=True)),
                       (lambda: first() + second(), grads(features=True, normals=True))):
        want = plain()
        counts = torch.count_nonzero(want[..., 0], dim=1)
        assert torch.all(counts >= 1000)
        ratio = off(got, want) / off(plain(), want)
        assert torch.all(ratio <= 1.3), ratio


@pytest.mark.parametrize("d,n", [(2, 2 ** 18 + 1), (7, 2 ** 20 - 3)])
def test_order_keeps_its_records_only(nat, d, n):
    """What an order holds on to is one record per point (the allocator rounds up to 512 bytes)."""
    enc, inp, _, _ = _setup(nat, d, 2, 4, n, 3)
    before = torch.cuda.memory_allocated()
    order = enc.order(inp)
    assert torch.cuda.memory_allocated() - before <= (16 if d <= 3 else 32) * n + 1024
    assert order is not None


@pytest.mark.parametrize("d", [3, 6])
def test_an_order_of_another_batch_is_refused(nat, d):
    n = 5000
    enc, inp, go, dpg = _setup(nat, d, 2, 4, n, 3)
    good = enc.order(inp)
    wide = torch.empty(2 * good.numel(), dtype=torch.uint8, device=DEV)
    wrong = [enc.order(_setup(nat, d, 2, 4, m, 3)[1]) for m in (n - 1, n + 1, 2 * n, n // 2)]
    wrong += [enc_.order(i) for enc_, i, _, _ in (_setup(nat, e, 2, 4, n, 3) for e in (2, 5))]
    wrong += [good.cpu(), good.view(torch.int8), good.float(), wide[16:16 + good.numel()], wide[::2], good[:-1]]
    weight = torch.randn(32, enc.output_width(), device=DEV)
    for order in wrong:
        inp.m_order = order
        for call in (lambda: enc.forward(inp), lambda: enc.forward_linear(inp, weight), lambda: enc.backward(inp, go),
                     lambda: enc.double_backward_from_positions(inp, dpg, go)):
            with pytest.raises(RuntimeError, match="spatial order does not belong"):
                call()
    whole = torch.empty(nat.lib.permuto_order_bytes(d, n), dtype=torch.uint8, device=DEV)   # filled by permuto_order_points
    whole[:good.numel()] = good
    want = enc.forward(nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, True, True))
    for order in (good, whole):
        inp.m_order = order
        assert torch.equal(enc.forward(inp), want)


@pytest.mark.parametrize("d,feat", [(2, 2), (3, 4), (6, 2)])
def test_rows_of_an_order_stay_inside_the_batch(nat, d, feat):
    """Whatever the buffer holds, no operation writes past the batch's rows."""
    n, room = 3001, 4096
    enc, inp, go, _ = _setup(nat, d, feat, 5, n, 9)
    gen = torch.Generator(device=DEV).manual_seed(4)
    for fill in (torch.full_like(enc.order(inp), 255),
                 torch.randint(0, 256, enc.order(inp).shape, device=DEV, generator=gen, dtype=torch.uint8)):
        inp.m_order = fill
        rows = torch.zeros((n + room, d), device=DEV)
        enc.backward(inp, go, positions_grad_out=rows[:n])
        torch.cuda.synchronize()
        assert torch.count_nonzero(rows[n:]) == 0
        assert enc.forward(inp).shape == (n, enc.output_width())
        torch.cuda.synchronize()


def test_a_call_without_room_for_an_order_runs_without_one(nat):
    """The order is an aid: a batch whose outputs fit runs whether or not the order fits beside them."""
    from permutohedral_encoding_b200 import PermutoEncoding
    n, levels = 2 ** 18 + 1, 16                                 # rows of 32 MB, records of 4 MB, scratch of 3 MB
    m = PermutoEncoding(3, 2 ** 10, levels, 2, np.ones(levels))
    pos = torch.rand(n, 3, device=DEV)
    go = torch.randn(n, 2 * levels, device=DEV)
    inp = nat.EncodingInput(m.lattice_values.detach(), pos, m.anneal_window, True, False)
    want, want_grad = m.lattice.forward(inp), m.lattice.backward(inp, go)[0]
    assert m.lattice.order(inp, nat.ORDER_TRAINING) is not None
    total = torch.cuda.get_device_properties(0).total_memory
    room, held = torch.empty(36 * 2 ** 20, dtype=torch.uint8, device=DEV), []

    def limit(extra):
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + extra) / total)

    try:
        limit(0)
        with pytest.raises(torch.cuda.OutOfMemoryError):   # nothing free but `room` and 2 MB
            while True:
                held.append(torch.empty(2 ** 21, dtype=torch.uint8, device=DEV))
        limit(2 ** 21)
        with pytest.raises(torch.cuda.OutOfMemoryError):
            m.lattice.order(inp)
        del room
        out = m(pos)
        out.backward(go)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        held.clear()
    assert torch.equal(out, want)
    assert torch.all((m.lattice_values.grad - want_grad).abs() <= 1e-4 * want_grad.abs().amax())


@pytest.mark.parametrize("share", [0.0, 0.2, 0.9])
@pytest.mark.parametrize("where", ["cuda", "cpu"])
def test_module_with_a_window(nat, share, where):
    """The module's calls with a mostly closed, a mostly open and a closed window, on a batch that is ordered
    when all levels are open: results as without an order."""
    from permutohedral_encoding_b200 import PermutoEncoding
    torch.manual_seed(8)
    n, levels = 2 ** 19 + 3, 16
    m = PermutoEncoding(3, 2 ** 10, levels, 2, np.geomspace(1.0, 1e-2, levels))
    with torch.no_grad():
        m.lattice_values.uniform_(-1, 1)
    window = torch.rand(levels) + 0.1
    window[int(levels * share):] = 0.0
    pos = torch.rand(n, 3, device=DEV, requires_grad=True)
    go, dpg = torch.randn(n, 2 * levels, device=DEV, requires_grad=True), torch.randn(n, 3, device=DEV)
    inp = nat.EncodingInput(m.lattice_values.detach(), pos.detach(), window.cuda(), True, True)
    want, (want_v, want_p) = m.lattice.forward(inp), m.lattice.backward(inp, go.detach())
    want_v2, want_g = m.lattice.double_backward_from_positions(inp, dpg, go.detach())

    def close(a, b):
        assert torch.all((a - b).abs() <= 1e-4 * b.abs().amax())

    w = window.to(where)
    with torch.no_grad():
        assert torch.equal(m(pos, w), want)
    out = m(pos, w)
    assert torch.equal(out, want)
    for a, b in zip(torch.autograd.grad(out, [m.lattice_values, pos], go), (want_v, want_p)):
        close(a, b)
    out = m(pos, w)
    (normal,) = torch.autograd.grad(out, pos, go, create_graph=True)
    got = torch.autograd.grad([out, normal], [m.lattice_values, go], [go.detach(), dpg])
    close(got[0], want_v + want_v2)
    close(got[1], want_g)
    close(torch.autograd.grad(m(pos.detach(), w), m.lattice_values, go)[0], want_v)


@pytest.mark.parametrize("zero", [True, False])
@pytest.mark.parametrize("n", [2 ** 21 + 4097, 2 ** 22 + 1025])
def test_buckets_of_levels_of_a_batch_of_several_chunks(nat, n, zero):
    """More points than one chunk of the sort, fewer and more than the table gradient is summed in order for:
    the features and, bucket by bucket as the data-parallel hook asks for them, both gradients, with the term
    of the concatenated points added once; onto a cleared table and onto one that the caller has cleared."""
    enc, inp, go, _ = _setup(nat, 3, 2, 7, n, 12, concat=True)
    enc.concat_positions_grad = True
    want = [enc.forward(inp), *enc.backward(inp, go)]
    magnitude = enc.backward(nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, True, False),
                             go.abs())[0]
    inp.m_order = enc.order(inp)
    assert torch.equal(enc.forward(inp), want[0])
    table = torch.full_like(want[1], float("nan")) if zero else torch.zeros_like(want[1])
    points = None
    for begin, end in ((0, 3), (3, 4), (4, 7)):
        got, points = enc.backward(inp, go, lattice_grad_out=table, level_begin=begin, level_end=end, zero=zero,
                                   positions_grad_out=points)
        assert got is table
    assert torch.all((table - want[1]).abs() <= 1e-4 * magnitude + 1e-6 * magnitude.amax())
    assert torch.all((points - want[2]).abs() <= 1e-5 * want[2].abs().amax())
    with pytest.raises(RuntimeError, match="level range"):
        enc.backward(inp, go, level_begin=4, level_end=3)


@pytest.mark.parametrize("n", [2 ** 20 + 3, 2 ** 22])
def test_table_gradient_against_float64(nat, n):
    """Summed in either sequence the table gradient is within 1e-5 (2-norm) of a float64 sum of the same
    addends, weight times gradient: k fp32 additions to one entry are off by about 2^-24 * sqrt(k) of what an
    entry holds, 6e-5 for a million and much less once a warp has merged its addends (measured: 0.7-6.5e-6)."""
    levels = 10
    enc, inp, go, _ = _setup(nat, 3, 2, levels, n, 31)
    inp = nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, torch.ones(levels, device=DEV), True, False)
    want = torch.zeros(inp.m_lattice_values.shape, dtype=torch.float64, device=DEV)
    for b in range(0, n, 2 ** 20):
        part = nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw[b:b + 2 ** 20], inp.m_anneal_window, True, False)
        r = enc.debug_lattice(part, want=("slots", "bary"))
        for l in range(levels):
            addends = r["bary"][:, l].double().unsqueeze(-1) * go[b:b + 2 ** 20, 2 * l:2 * l + 2].double().unsqueeze(1)
            want[l].index_add_(0, r["slots"][:, l].reshape(-1).long(), addends.reshape(-1, 2))
    for inp.m_order in (None, enc.order(inp)):
        assert (enc.backward(inp, go)[0].double() - want).norm() <= 1e-5 * want.norm()


def test_an_ordered_step_can_be_replayed_from_a_cuda_graph(nat):
    """The sort, its early launches among them, and both backward kernels are captured; a replay sorts the
    positions that are there then."""
    from permutohedral_encoding_b200 import PermutoEncoding
    torch.manual_seed(6)
    n, levels = 2 ** 19 + 5, 16
    m = PermutoEncoding(3, 2 ** 12, levels, 2, np.geomspace(1.0, 1e-2, levels))
    with torch.no_grad():
        m.lattice_values.uniform_(-1, 1)
    first, pos = torch.rand(n, 3, device=DEV), torch.rand(n, 3, device=DEV) - 0.5
    static, go = first.clone().requires_grad_(True), torch.randn(n, 2 * levels, device=DEV)
    inp = nat.EncodingInput(m.lattice_values.detach(), pos, m.anneal_window, True, True)
    assert m.lattice.order(inp, nat.ORDER_POSITIONS) is not None
    want = [m.lattice.forward(inp), *m.lattice.backward(inp, go)]

    def step():
        m.lattice_values.grad = static.grad = None
        out = m(static)
        out.backward(go)
        return out

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    graph.replay()
    with torch.no_grad():
        static.copy_(pos)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[0])
    for a, b in zip((m.lattice_values.grad, static.grad), want[1:]):
        assert torch.all((a - b).abs() <= 1e-4 * b.abs().amax())


@pytest.mark.parametrize("d,feat,levels,n", [
    (3, 2, 1, 700), (3, 2, 33, 17), (2, 2, 24, 4111), (4, 4, 11, 2 ** 15 + 1), (7, 8, 130, 300),   # strands of one point and
    # more, blocks with idle threads, more levels than a block has threads; below: either side of the lines between
    # one and two vertices per remainder
    (3, 2, 6, 3 * 2 ** 17 - 1), (3, 2, 6, 3 * 2 ** 17), (4, 2, 5, 3 * 2 ** 18 - 1), (4, 2, 5, 3 * 2 ** 18),
    (5, 2, 4, 3 * 2 ** 18), (5, 2, 4, 3 * 2 ** 19), (6, 2, 5, 2 ** 18 + 3)])
def test_table_gradients_of_strands(nat, d, feat, levels, n):
    """Every form of the ordered table gradient against the unordered kernels: the same fp32 addends in another
    sequence, with and without merging, with levels closed; bound as above."""
    enc, inp, go, dpg = _setup(nat, d, feat, levels, n, 5 * d + levels)
    inp = nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, True, False)

    def run(order):
        inp.m_order = order
        return [enc.backward(inp, go)[0], enc.double_backward_from_positions(inp, dpg, go, need_grad_grad_features=False)[0]]

    plain, order = run(None), enc.order(inp)
    magnitude = enc.backward(nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, True, False), go.abs())[0]
    for enc.aggregate_collisions in (True, False) if n < 2 ** 16 else (True,):
        for a, b, m in zip(plain, run(order), (magnitude, plain[1].abs().amax().expand_as(plain[1]))):
            assert torch.all((a - b).abs() <= 1e-4 * m + 1e-6 * m.amax())


@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("d,levels,n,concat", [(3, 24, 2 ** 15 + 5, False), (2, 9, 31, True), (3, 33, 4111, True), (3, 1, 700, False)])
def test_both_gradients_in_one_walk(nat, d, levels, n, concat, half):
    """The position gradient that comes with the ordered table gradient: batches of points that end inside a
    strand, closed levels, concatenated points, accumulation onto a given gradient, level ranges.  The same fp32
    terms summed level by level: bound as for other groupings of the levels."""
    enc, inp, go, _ = _setup(nat, d, 2, levels, n, levels, concat=concat, half=half)
    enc.concat_positions_grad = True
    plain = enc.backward(inp, go)
    magnitude = enc.backward(nat.EncodingInput(inp.m_lattice_values, inp.m_positions_raw, inp.m_anneal_window, True, False), go.abs())[0]
    inp.m_order = enc.order(inp)
    got = enc.backward(inp, go)
    assert torch.all((got[0] - plain[0]).abs() <= 1e-4 * magnitude + 1e-6 * magnitude.amax())
    assert torch.all((got[1] - plain[1]).abs() <= 1e-5 * plain[1].abs().amax())
    table, points = torch.zeros_like(got[0]), torch.ones_like(got[1])
    for begin, end in ((0, levels // 2), (levels // 2, levels)):
        enc.backward(inp, go, lattice_grad_out=table, level_begin=begin, level_end=end, positions_grad_out=points)
    assert torch.all((table - plain[0]).abs() <= 1e-4 * magnitude + 1e-6 * magnitude.amax())
    assert torch.all((points - 1 - plain[1]).abs() <= 1e-5 * plain[1].abs().amax() + 1e-6)
