"""The norm behind the scans in 16-byte pieces and the gates' maximum over blocks of tokens, at the edges of their pieces."""
import pytest
import torch

from tests import kernel_refs as refs

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("part", [8, 64, 72, 128, 136, 256, 264, 512, 520, 2048, 2056, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("gate,first,extras", [("sigmoid", False, "denominator"), ("silu", True, "skip"), ("silu", False, "")])
def test_gated_group_norm_pieces(part, gate, first, extras):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(part)
    n, parts = 5, 3
    c, heads = parts * part, 3
    y, wide = torch.randn(n, c, generator=g, device=DEV), torch.randn(n, 2 * c + 8, generator=g, device=DEV).bfloat16()
    weight = (1 + 0.2 * torch.randn(c, generator=g, device=DEV)).bfloat16()
    more = {}
    if extras == "denominator":
        more = dict(nq=torch.randn(n, heads, generator=g, device=DEV), floor=torch.rand(n, heads, generator=g, device=DEV), floor_add=1e-6)
    elif extras == "skip":
        more = dict(skip=torch.randn(heads, generator=g, device=DEV), skip_x=wide[:, c + 8:])
    for gates in (wide[:, :c], wide[:, 1:c + 1]):   # 16-byte places, and places that the scalar kernel takes
        out, want = (torch.empty(n, c, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        ops.gated_group_norm(y, gates, weight, 1e-5, out, parts, heads, gate, first, **more)
        refs.gated_group_norm(y, gates, weight, 1e-5, want, parts, heads, gate, first, **more)
        # both sides round one float32 number to bfloat16 and so are neighbours at most; neighbours (8 significant bits) are up to
        # 2^-7 of the value apart
        assert float(((out.double() - want.double()).abs() / (want.double().abs() + 1e-3)).max()) <= 2 ** -7


@pytest.mark.parametrize("lengths", [(1,), (255, 256, 257), (2047, 2048, 2049), (5000, 31)])
def test_stabilized_gates_over_blocks_of_tokens(lengths):
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(len(lengths))
    heads, n = 3, sum(lengths)
    cu, slots = [0], [2, -1, 0][:len(lengths)]
    for length in lengths:
        cu.append(cu[-1] + length)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pre, bias = 6 * torch.randn(n, 2 * heads, generator=g, device=DEV), torch.randn(2 * heads, generator=g, device=DEV)
    start = torch.rand(4, 20, generator=g, device=DEV)
    results = []
    for fn in (ops.stabilized_gates, refs.stabilized_gates):
        state, trio = start.clone(), [torch.empty(n, heads, device=DEV) for _ in range(3)]
        fn(pre, bias, 15.0, ints(cu), ints(slots), state, 7, heads, *trio)
        results.append((state, *trio))
    # m is a sum of up to a few dozen log gates of size up to 15 before a larger one takes over: 2^-24 x 15 x a few dozen
    for got, want in zip(*results):
        assert float(((got.double() - want.double()).abs() / (1 + want.double().abs())).max()) < 3e-5


@pytest.mark.parametrize("pieces", [[1] * 300, [255, 256, 257, 2048, 1], [7, 2049, 8, 9, 2040]])
def test_stabilized_gates_do_not_depend_on_the_cut(pieces):
    """The maximum is one chain of additions and maxima in the tokens' order: bit for bit the same numbers however a sequence is cut,
    and every token is decayed with the very maximum that the token before it was scaled by."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(len(pieces))
    heads, n = 3, sum(pieces)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pre, bias = 2 * torch.randn(n, 2 * heads, generator=g, device=DEV), torch.tensor([0.0] * heads + [3.0] * heads, device=DEV)
    results = []
    for cut in ([n], pieces):
        state, trio, at = torch.zeros(1, heads, device=DEV), [torch.empty(n, heads, device=DEV) for _ in range(3)], 0
        for length in cut:
            here = slice(at, at + length)
            ops.stabilized_gates(pre[here], bias, 15.0, ints([0, length]), ints([0]), state, 0, heads, *(t[here] for t in trio))
            at += length
        results.append((state, *trio))
    for whole, cut in zip(*results):
        assert torch.equal(whole, cut)


def test_gates_far_below_zero():
    """sigmoid and silu as float32 forms them, down to where e^-z overflows (z = -88.7): nothing becomes zero before that."""
    from qwenforge_b200 import ops
    n, c, taps = 64, 64, 4
    z = torch.linspace(-88.5, -60, n, device=DEV).bfloat16()[:, None].expand(n, c).contiguous()
    want = z.double() * torch.sigmoid(z.double())
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    weight = torch.zeros(c, taps, device=DEV)
    weight[:, -1] = 1.0                                        # only the newest input counts
    for single in (False, True):   # one sequence of n tokens, n sequences of one token
        cu, seqs = (list(range(n + 1)), list(range(n))) if single else ([0, n], [0] * n)
        state, got = torch.zeros(n, (taps - 1) * c, device=DEV), torch.empty(n, c, dtype=torch.bfloat16, device=DEV)
        ops.causal_conv_silu(z, weight, None, ints(cu), ints(seqs), ints(list(range(n))[:len(cu) - 1]), state, 0, got, single=single)
        assert float(((got.double() - want) / want).abs().max()) <= 2 ** -8
    ones, out = torch.ones(n, c, device=DEV), torch.empty(n, c, dtype=torch.bfloat16, device=DEV)
    for gate, size in (("silu", want), ("sigmoid", torch.sigmoid(z.double()))):
        ops.gated_group_norm(ones, z, torch.ones(c, dtype=torch.bfloat16, device=DEV), 0.0, out, 1, 1, gate, False)
        # (a sigmoid below 2^-126 has fewer bits: 2^-149 is its unit, and a bfloat16 below 2^-126 has 2^-133)
        assert float(((out.double() - size).abs() / (size.abs() * 2 ** -7 + 2.0 ** -133)).max()) <= 1


def test_silu_behind_the_convolution():
    """Taps of zero and one leave the input: silu of float32 numbers over their whole range. Two roundings of the exponential (2 ulp)
    count at most |z| / (1 + e^z) <= 1 each, then one of the sum and one of the quotient."""
    from qwenforge_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(5)
    x = torch.randn(64, 4096, generator=g, device=DEV) * torch.logspace(-6, 1.4, 64, device=DEV)[:, None]
    x[:, 0] = 0.0                                              # (what is not finite stays in its own token: no tap in front of it)
    odd = torch.tensor([0.0, -0.0, 100.0, -100.0, -88.0, float("inf"), float("nan")], device=DEV)
    n, c = x.shape
    cu, slots = torch.tensor([0, n], dtype=torch.int32, device=DEV), torch.tensor([-1], dtype=torch.int32, device=DEV)
    seq, taps = torch.zeros(n, dtype=torch.int32, device=DEV), torch.tensor([[0.0, 1.0]], device=DEV).repeat(c, 1)
    last = x.clone()
    last[-1, :odd.numel()] = odd
    out, state = torch.empty_like(x), torch.zeros(1, c, device=DEV)
    ops.causal_conv_silu(last, taps, None, cu, seq, slots, state, 0, out)
    z = last.double()
    want, got = z / (1 + torch.exp(-z)), out.double()
    fine = torch.isfinite(want) & (z.abs() < 80)
    assert bool(((got - want).abs()[fine] <= 4 * 2.0 ** -23 * want.abs()[fine]).all())
    row = out[-1, :odd.numel()].tolist()
    assert row[0] == row[1] == 0 and row[2] == 100 and abs(row[3]) < 1e-35 and abs(row[4]) < 1e-35 and row[5] == float("inf") and row[6] != row[6]


def test_silu_has_the_bits_of_the_division():
    """Every float32 number through the convolution's silu, against 1 + e^-z and z / that as CUDA rounds them: the same bits; results
    below 2^-126 are one unit (2^-149) apart at most. In runs of tokens, and a sample token by token."""
    from qwenforge_b200 import ops
    n = c = 8192
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    cu, seq, state = ints([0, n]), torch.zeros(n, dtype=torch.int32, device=DEV), torch.zeros(1, c, device=DEV)
    last = torch.tensor([[0.0, 1.0]], device=DEV).repeat(c, 1)                # only the newest input counts
    offsets = torch.arange(n * c, dtype=torch.int32, device=DEV)
    wrong = torch.zeros(2, dtype=torch.int64, device=DEV)
    out = torch.empty(n, c, device=DEV)
    for chunk in range(64):
        x = (offsets + (chunk * n * c - (1 << 31))).view(torch.float32).view(n, c)
        x = torch.where(torch.isfinite(x), x, torch.zeros_like(x)) + 0.0   # (a number that is not finite would reach the next token)
        want = x / (torch.exp(-x) + 1.0)
        for taps in ((last, last[:, 1:].contiguous()) if chunk % 16 == 0 else (last,)):
            ops.causal_conv_silu(x, taps, None, cu, seq, ints([-1]), state, 0, out)
            small = want.abs() < 2.0 ** -126
            wrong[0] += (~small & (out != want)).sum()
            wrong[1] += (small & ((out - want).abs() > 2.0 ** -149)).sum()
    assert wrong.tolist() == [0, 0]


@pytest.mark.parametrize("gate,first", [("sigmoid", False), ("silu", False), ("silu", True)])
def test_gates_of_the_norm_have_the_bits_of_the_division(gate, first):
    """Every bfloat16 gate, in pieces of eight columns and (rows that no 16-byte load can address) number by number with `/`."""
    from qwenforge_b200 import ops
    values = torch.arange(-32768, 32768, dtype=torch.int32, device=DEV).short().view(torch.bfloat16)
    values = values[torch.isfinite(values) & (values.abs() < 1e18)].repeat_interleave(8).view(-1, 8)   # (a row per gate: `first` squares it)
    n = values.shape[0]
    off = torch.zeros(n, 16, dtype=torch.bfloat16, device=DEV)
    off[:, 1:9] = values
    g = torch.Generator(device=DEV).manual_seed(1)
    # one number a row, so that the sum of squares is the same in any order
    y, weight = torch.zeros(n, 8, device=DEV), torch.randn(8, generator=g, device=DEV).bfloat16()
    y.scatter_(1, torch.randint(0, 8, (n, 1), generator=g, device=DEV), torch.randn(n, 1, generator=g, device=DEV))
    results = []
    for gates in (values, off[:, 1:9]):
        out = torch.empty(n, 8, dtype=torch.bfloat16, device=DEV)
        ops.gated_group_norm(y, gates, weight, 1e-5, out, 1, 1, gate, first)
        results.append(out)
    assert torch.equal(*results) and bool(torch.isfinite(results[0]).all())
