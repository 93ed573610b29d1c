"""The element-wise network operators' 16-byte paths give the bits of their
element-wise paths (taken when an address is off by one element), over lengths
with and without a remainder and values that include infinities, NaN and zeros of
both signs.  The bias gradient, whose summation order differs between the two, is
checked against float64 (FP32 sums of n terms: n 2^-24 of the sum of magnitudes)."""
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ops(wt_lib):
    from windtunnel.net import Ops
    return Ops()


def shifted(t):
    """A copy of t whose address is one element past an aligned one."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    out = flat[1:].view(t.shape)
    out.copy_(t)
    return out


def values(shape, dtype, seed, special=True):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randn(shape, generator=g, device="cuda")
    if special and t.numel() >= 40:
        f = t.view(-1)
        f[3], f[9], f[17], f[33], f[35] = float("inf"), float("nan"), -0.0, 0.0, float("-inf")
    return t.to(dtype)


def bits(t):
    return t.contiguous().view(torch.int16 if t.dtype == torch.bfloat16 else torch.int32)


def both(call, ins, out):
    """call on aligned tensors and on shifted ones: equal bits."""
    o1, o2 = out.clone(), shifted(out)
    call(ins, o1)
    call([None if t is None else shifted(t) for t in ins], o2)
    torch.cuda.synchronize()
    assert torch.equal(bits(o1), bits(o2))


@pytest.mark.parametrize("shape", [(1, 1, 1, 1, 8), (2, 3, 5, 1, 16), (3, 2, 1, 7, 24), (1, 4, 3, 2, 4)])
def test_pooling_and_upsampling(ops, shape):
    b, d, h, w, c = shape
    fine = (b, 2 * d, 2 * h, 2 * w, c)
    bf, f32 = torch.bfloat16, torch.float32
    both(lambda i, o: ops.pool2(i[0], o), [values(fine, bf, 1)], torch.empty(shape, dtype=bf, device="cuda"))
    both(lambda i, o: ops.up2(i[0], o), [values(shape, bf, 2)], torch.empty(fine, dtype=bf, device="cuda"))
    both(lambda i, o: ops.pool2_backward(i[0], o), [values(shape, f32, 3)], torch.empty(fine, dtype=f32, device="cuda"))
    both(lambda i, o: ops.up2_backward(i[0], o), [values(fine, f32, 4)], torch.empty(shape, dtype=f32, device="cuda"))


@pytest.mark.parametrize("n", [1, 7, 8, 40, 2049, 4096 * 8 + 3])
def test_elementwise(ops, n):
    bf, f32 = torch.bfloat16, torch.float32
    out = torch.empty(n, dtype=bf, device="cuda")
    a, b, g, g2, act = values(n, bf, 1), values(n, bf, 2), values(n, f32, 3), values(n, f32, 4), values(n, bf, 5)
    both(lambda i, o: ops.add(i[0], i[1], o), [a, b], out)
    for second in (None, g2):
        for mask in (None, act):
            both(lambda i, o: ops.grad_to_bf16(i[0], i[1], i[2], o), [g, second, mask], out)
    state = [values(n, f32, 6, False), values(n, f32, 7, False), values(n, f32, 8, False).abs()]  # p, m, v
    two = [[t.clone() for t in state], [shifted(t) for t in state]]
    copies = [torch.empty(n, dtype=bf, device="cuda"), shifted(torch.empty(n, dtype=bf, device="cuda"))]
    for (p, m, v), pb, grad in zip(two, copies, (g.nan_to_num(1.0, 2.0, -2.0), shifted(g.nan_to_num(1.0, 2.0, -2.0)))):
        ops.adam(p, grad, m, v, pb, 1e-2, 3)
    for x, y in zip([*two[0], copies[0]], [*two[1], copies[1]]):
        assert torch.equal(bits(x), bits(y))


@pytest.mark.parametrize("rows", [1, 33, 70000])
def test_loss_gradient(ops, rows):
    pred, target = values((rows, 8), torch.bfloat16, 1, False), values((rows, 4), torch.float32, 2, False)
    mask = (values(rows, torch.float32, 3, False) > 0).float()
    losses = []

    def call(i, o):
        loss = torch.zeros(1, dtype=torch.float64, device="cuda")
        ops.mse(i[0], i[1], mask, 7.0, o, loss)
        losses.append(loss)

    both(call, [pred, target], torch.empty((rows, 8), dtype=torch.bfloat16, device="cuda"))
    want = (mask[:, None].double() * (pred[:, :4].double() - target.double()) ** 2).sum()
    for loss in losses:
        assert abs(float(loss) - float(want)) <= 4e-7 * float(want)  # products formed in FP32


@pytest.mark.parametrize("c", [1, 4, 8, 64, 256])
@pytest.mark.parametrize("rows", [1, 511, 40001])
def test_bias_gradient(ops, rows, c):
    dy = values((rows, c), torch.bfloat16, rows + c, False)
    want, scale = dy.double().sum(0), dy.double().abs().sum(0)
    for t in (dy, shifted(dy)):
        db = torch.empty(c, device="cuda")
        ops.bias_grad(t, db)
        assert bool(((db.double() - want).abs() <= rows * 2.0 ** -24 * scale + 1e-30).all())
