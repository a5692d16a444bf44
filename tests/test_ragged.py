"""GPU: sizes whose rows are no multiple of 16 bytes, at the edges of the tiles and vectors of the kernels that take them:
products with element-wise epilogues (one- and two-CTA kernels, split contraction, addend and mask), the operand packing
with its mask and column sums, and the cross-entropy rows.  Bounds: one 16-bit rounding of the result (2^-11 / 2^-8 of
its size) plus fp32 accumulation."""
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _close(got, want, dtype, terms=1):
    err = (got.double() - want).abs()
    # one rounding of the result, and fp32 sums of `terms` products of values of about one
    bound = EPS[dtype] * want.abs() + 2.0 ** -22 * terms + 2.0 ** -24
    assert (err <= 1.01 * bound).all(), (err - bound).max().item()


# (M, N, K): one tile and its edges, several tiles, the pair kernel, split contractions; N odd or even without being 8k
PRODUCTS = [(1, 1, 8), (31, 33, 64), (128, 127, 72), (129, 257, 128), (300, 250, 640), (640, 1001, 4096), (2600, 1290, 256),
            (5000, 2050, 128)]


@pytest.mark.parametrize("m,n,k", PRODUCTS)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("form", ["plain", "bias_relu", "addend_mask"])
def test_products_with_unaligned_output_rows(m, n, k, dtype, form):
    from tritonformer_b200 import linear as L
    torch.manual_seed(m + n + k)
    a = torch.randn(m, k, device="cuda").to(dtype)
    w = (torch.randn(n, k, device="cuda") * k ** -0.5).to(dtype)  # applied transposed: its rows are aligned
    want = a.double() @ w.double().t()
    extra = {}
    if form == "bias_relu":
        bias = torch.randn(n, device="cuda").to(dtype)
        want, extra = (want + bias.double()).clamp_min(0.0), {"bias": bias, "relu": True}
    elif form == "addend_mask":
        add, mask = (torch.randn(m, n, device="cuda").to(dtype) for _ in range(2))
        want, extra = torch.where(mask > 0, want + add.double(), 0.0), {"addend": add, "mask": mask}
    calls = []
    L.PROFILE = calls
    try:
        got = L.gemm(a, k, 1, w, 1, k, m, n, k, **extra)
    finally:
        L.PROFILE = None
    assert calls[0]["path"] == 1  # the tcgen05 kernels
    _close(got, want, dtype, terms=k ** 0.5)


@pytest.mark.parametrize("rows,cols", [(1, 1), (7, 3), (33, 255), (64, 257), (1000, 1477), (4099, 9)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("offset", [0, 1, 5])
def test_grad_rows(rows, cols, dtype, offset):
    """The mask, the packing and the column sums, from every kind of base address."""
    from tritonformer_b200 import _lib as L
    dy = torch.randn(rows * cols + offset, device="cuda").to(dtype)[offset:].view(rows, cols)
    act = torch.randn(rows * cols + offset, device="cuda").to(dtype)[offset:].view(rows, cols)
    ld = -(-cols // 8) * 8
    dz = torch.full((rows, ld), 7.0, device="cuda", dtype=dtype)
    sums = torch.empty(cols, device="cuda", dtype=dtype)
    n = L.lib.tfb_colsum_partials(rows, cols)
    partials = torch.empty(n, cols, device="cuda")
    L.check(L.lib.tfb_grad_rows(dy.data_ptr(), act.data_ptr(), dz.data_ptr(), sums.data_ptr(), partials.data_ptr(), n, rows,
                                cols, cols, cols, ld, L.dtype_code(dtype), L.stream_ptr(dy.device)))
    want = torch.where(act > 0, dy, torch.zeros_like(dy))
    assert torch.equal(dz[:, :cols], want) and not dz[:, cols:].any()
    _close(sums, want.double().sum(0), dtype, terms=rows)
    L.check(L.lib.tfb_grad_rows(dy.data_ptr(), None, dz.data_ptr(), None, None, 0, rows, cols, cols, 0, ld,
                                L.dtype_code(dtype), L.stream_ptr(dy.device)))
    assert torch.equal(dz[:, :cols], dy)


@pytest.mark.parametrize("cols", [247, 248, 249, 495, 496, 497])
@pytest.mark.parametrize("rows", [1, 31, 1300])
def test_grad_rows_at_the_edges_of_a_warps_columns(rows, cols):
    """A warp writes 248 columns; what it reads beside them is its neighbour's first vector, or nothing."""
    for offset in range(8):
        test_grad_rows(rows, cols, torch.float16, offset)


@pytest.mark.parametrize("rows,cols", [(9472, 9), (9480, 247), (9472, 248), (9473, 249), (4736, 495), (4749, 496), (4737, 497), (1200, 2049)])
def test_grad_rows_with_several_rows_a_warp(rows, cols):
    """From two misaligned rows per warp on: the kernel whose lanes take the misaligned halves from their neighbours."""
    for offset in range(8):
        test_grad_rows(rows, cols, torch.float16, offset)
    test_grad_rows(rows, cols, torch.bfloat16, 3)


@pytest.mark.parametrize("rows,cols,pitch,offset,shifted", [
    (9472, 249, 249, 0, True), (9472, 249, 256, 0, False), (9472, 249, 256, 1, True), (9472, 256, 256, 0, False),
    (4735, 249, 249, 0, False), (64, 65, 65, 0, False)])
@pytest.mark.parametrize("masked", [False, True])
def test_only_misaligned_rows_are_shifted(rows, cols, pitch, offset, shifted, masked):
    """Aligned rows, and misaligned ones of which a warp has less than two, keep the kernel that loads them as they lie."""
    from torch.profiler import ProfilerActivity, profile
    from tritonformer_b200 import _lib as L
    src = torch.randn(rows * pitch + 8, device="cuda").half()[offset:]
    dz = torch.empty(rows, -(-cols // 8) * 8, device="cuda", dtype=torch.half)
    call = (src.data_ptr(), src.data_ptr() if masked else None, dz.data_ptr(), None, None, 0, rows, cols, pitch, pitch, dz.shape[1],
            L.dtype_code(torch.half), L.stream_ptr(dz.device))
    L.check(L.lib.tfb_grad_rows(*call))
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        L.check(L.lib.tfb_grad_rows(*call))
        torch.cuda.synchronize()
    names = [e.key for e in p.key_averages() if "grad_rows" in e.key]
    assert len(names) == 1 and ("grad_rows_kernel<__half>" in names[0]) != shifted, names
    want = src[:rows * pitch].view(rows, pitch)[:, :cols]
    assert torch.equal(dz[:, :cols], want.clamp_min(0.0) if masked else want)


@pytest.mark.parametrize("cols", [1, 7, 9, 2047, 2049, 50257])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_lm_loss_of_an_odd_vocabulary(cols, dtype):
    from tritonformer_b200.crossentropy import lm_loss
    torch.manual_seed(cols)
    b, t = 2, 9
    logits = torch.randn(b, t, cols, device="cuda").to(dtype).requires_grad_(True)
    labels = torch.randint(0, cols, (b, t), device="cuda")
    ref = logits.detach().double().requires_grad_(True)
    want = torch.nn.functional.cross_entropy(ref[:, :-1].reshape(-1, cols), labels[:, 1:].reshape(-1))
    loss = lm_loss(logits, labels)
    assert abs(loss.item() - want.item()) <= 1e-5 * max(1.0, abs(want.item()))
    (loss * 16.0).backward()
    (want * 16.0).backward()
    # exp2f of an fp32 difference: a few 1e-6 of the probability, then one rounding (or half a subnormal step)
    err = (logits.grad.double() - ref.grad).abs()
    assert (err <= (EPS[dtype] + 1e-5) * ref.grad.abs() + 1e-6 + 2.0 ** -25).all()


@pytest.mark.parametrize("table_dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("dtype,hd,t", [(torch.float16, 64, 192), (torch.bfloat16, 128, 2560)])
def test_alibi_table_penalty_is_the_tables_entry(dtype, hd, t, table_dtype):
    """Queries and keys of zero leave the scores to the bias alone, so an entry that is rounded otherwise than the table's
    shows: the fp16 distances above 2048 and the bf16 ones above 256 are themselves rounded."""
    from tritonformer_b200.attention import BiasedCausalAttention
    from tritonformer_b200.transformer import generate_alibi_mask
    h = 6  # slopes that are no powers of two among them
    table = generate_alibi_mask(t, h, device="cuda", dtype=table_dtype)[0]
    q = torch.zeros(1, h, t, hd, device="cuda", dtype=dtype)
    v = (torch.rand(1, h, t, hd, device="cuda") * 2 - 1).to(dtype)
    out = BiasedCausalAttention.apply(q, q, v, table)
    want = torch.softmax(table.double(), -1) @ v[0].double()
    # |v| <= 1 and the probabilities sum to one: half a unit of the 16-bit type for the probabilities, half for the output,
    # and 7.5e-5 for the cubic exponential (twice: numerator and row sum)
    tol = (2.0 ** -10 if dtype is torch.float16 else 2.0 ** -8) + 2e-4
    assert (out[0].double() - want).abs().max().item() < tol


@pytest.mark.parametrize("heads,t,hd", [(300, 64, 64), (333, 128, 128), (333, 128, 32), (150, 192, 64), (120, 384, 128), (90, 640, 64)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_attention_backward_with_several_items_per_sm(heads, t, hd, dtype):
    """More (key tile, head) items than SMs, walks of one tile among them: a CTA goes on to the blocks that have not started."""
    from tritonformer_b200.attention import CausalAttention
    torch.manual_seed(heads + t)
    q, k, v = (torch.randn(1, heads, t, hd, device="cuda").to(dtype).requires_grad_() for _ in range(3))
    g = torch.randn(1, heads, t, hd, device="cuda").to(dtype)
    got = torch.autograd.grad(CausalAttention.apply(q, k, v), (q, k, v), g)
    qd, kd, vd = (x.detach().double().requires_grad_() for x in (q, k, v))
    s = (qd @ kd.transpose(-1, -2)) / hd ** 0.5
    s = s.masked_fill(~torch.ones(t, t, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.autograd.grad(torch.softmax(s, -1) @ vd, (qd, kd, vd), g.double())
    for a, b in zip(got, want):
        # per head, in the 2-norm: P, dS, the saved output (in delta) and the gradient itself are each rounded to 16 bits
        err = (a.double() - b).flatten(2).norm(dim=2) / b.flatten(2).norm(dim=2)
        assert err.max().item() < 4 * EPS[dtype]
