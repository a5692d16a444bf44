"""GPU: every plan of the one-wave GEMM kernel (tile width, CTA pairs, workers that share the contraction) and the persistent
kernels behind it, chosen through the tuning switch, each with the plan that ran asserted.  Bounds as in test_ragged.py, with
the K / 16 steps of the contraction as the terms: each may cut a unit in the last place off an fp32 sum of about one."""
import pytest
import torch

import test_fused
from test_ragged import _close

pytestmark = pytest.mark.gpu
NO_ONE_WAVE = 128


@pytest.fixture
def switches():
    from tritonformer_b200 import _lib

    def set_switches(value):
        torch.cuda.synchronize()
        _lib.lib.tfb_debug_set(4, value)

    yield set_switches
    set_switches(0)


def _operands(m, n, k, layout, dtype=torch.float16):
    """(a, a_sm, a_sk, b, b_sk, b_sn, a in fp64, b in fp64); layout: which of A and B is contiguous along M / N."""
    gen = torch.Generator(device="cuda").manual_seed(m + 3 * n + 5 * k)
    r = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    a = r(k, m).to(dtype) if layout[0] == "m" else r(m, k).to(dtype)
    b = (r(k, n) * k ** -0.5).to(dtype) if layout[1] == "n" else (r(n, k) * k ** -0.5).to(dtype)
    a_str = (1, m) if layout[0] == "m" else (k, 1)
    b_str = (n, 1) if layout[1] == "n" else (1, k)
    return (a, *a_str, b, *b_str, a.double().t() if layout[0] == "m" else a.double(),
            b.double() if layout[1] == "n" else b.double().t())


def _check_all_epilogues(m, n, k, layout, dtype=torch.float16):
    from tritonformer_b200 import linear as L
    *args, ad, bd = _operands(m, n, k, layout, dtype)
    want, terms = ad @ bd, k / 16
    gen = torch.Generator(device="cuda").manual_seed(1)
    bias, add, mask = (torch.randn(*s, device="cuda", generator=gen).to(dtype) for s in ((n,), (m, n), (m, n)))
    first = L.gemm(*args, m, n, k)
    _close(first, want, dtype, terms)
    assert torch.equal(first, L.gemm(*args, m, n, k))  # the order of the sums does not depend on timing
    _close(L.gemm(*args, m, n, k, bias=bias, relu=True), (want + bias.double()).clamp_min(0.0), dtype, terms)
    _close(L.gemm(*args, m, n, k, mask=mask), torch.where(mask > 0, want, 0.0), dtype, terms)
    full = torch.where(mask > 0, (want + bias.double()).clamp_min(0.0) + add.double(), 0.0)
    _close(L.gemm(*args, m, n, k, bias=bias, relu=True, addend=add, mask=mask), full, dtype, terms)
    into = add.clone()
    L.gemm(*args, m, n, k, out=into, accumulate=True)
    _close(into, want + add.double(), dtype, terms)
    # an output whose rows no box can describe
    odd = torch.full((m, n + 1), 7.0, device="cuda", dtype=dtype)
    from tritonformer_b200 import _lib
    a, a_sm, a_sk, b, b_sk, b_sn = args
    _lib.check(_lib.lib.tfb_gemm_fused(a.data_ptr(), b.data_ptr(), odd.data_ptr(), bias.data_ptr(), add.data_ptr(), n,
                                       mask.data_ptr(), n, m, n, k, a_sm, a_sk, b_sk, b_sn, n + 1, 1,
                                       _lib.dtype_code(dtype), None, 0, _lib.stream_ptr(a.device), None))
    _close(odd[:, :n], full, dtype, terms)
    assert bool((odd[:, n] == 7.0).all())


PLANS = [(bn, pair, split) for bn, pair in ((64, 0), (128, 0), (128, 1), (192, 1), (256, 1)) for split in (1, 2, 4, 8)
         if split <= (4 if pair else 8)]


@pytest.mark.parametrize("bn,pair,split", PLANS)
@pytest.mark.parametrize("layout", ["kn", "kk", "mn", "mk"])
@pytest.mark.parametrize("m,n,k", [(152, 200, 1096), (264, 392, 584), (8, 16, 520), (1, 8, 512)])
def test_one_wave_plans(bn, pair, split, layout, m, n, k, switches):
    from tritonformer_b200 import _lib
    if layout[0] == "m" and m % 8:
        pytest.skip("A contiguous along M needs whole vectors of M")
    code = 1 + bn // 64 * 2 + pair + 16 * split
    switches(code << 16)
    tiles = -(-m // (256 if pair else 128)) * -(-n // bn)
    if pair and (m <= 128 or n < 64):
        assert _lib.lib.tfb_debug_gemm_plan(m, n, k, int(layout[1] == "n")) == 0  # not a plan of this product
        return
    if tiles * split * (1 + pair) > 128:  # (clusters leave a few of the 148 SMs idle)
        pytest.skip("more CTAs than certainly run at the same time")
    assert _lib.lib.tfb_debug_gemm_plan(m, n, k, int(layout[1] == "n")) == code
    _check_all_epilogues(m, n, k, layout)


@pytest.mark.parametrize("bn,pair,split", [(64, 0, 8), (128, 0, 1), (192, 1, 2), (256, 1, 4)])
def test_one_wave_plans_bf16(bn, pair, split, switches):
    switches((1 + bn // 64 * 2 + pair + 16 * split) << 16)
    _check_all_epilogues(264, 392, 584, "mn", torch.bfloat16)


def test_whole_tiles_only(switches):
    from tritonformer_b200 import _lib
    assert _lib.lib.tfb_debug_gemm_plan(128, 128, 8192, 1) // 16 > 1  # shares the contraction by default
    switches(1)
    assert _lib.lib.tfb_debug_gemm_plan(128, 128, 8192, 1) // 16 == 1
    _check_all_epilogues(128, 128, 8192, "kn")


@pytest.mark.parametrize("shape", test_fused.STREAM_K_SHAPES)
@pytest.mark.parametrize("layout", ["weight_grad", "forward", "input_grad"])
def test_persistent_kernels(shape, layout, switches):
    """The shapes of the stream-K test on the kernels that it is about, with the one-wave kernel out of the way."""
    from tritonformer_b200 import _lib
    switches(NO_ONE_WAVE)
    assert _lib.lib.tfb_debug_gemm_plan(*shape, 1) == 0
    test_fused.test_stream_k_gemm_matches_fp32_and_is_deterministic(shape, layout)


@pytest.mark.parametrize("m,n,k", [(64, 25152, 1024), (64, 25153, 1024), (128, 20000, 1088), (1, 19001, 2048)])
def test_persistent_split_that_is_reached_by_default(m, n, k):
    """One tile row over more columns than one wave of tiles: the contraction of a tile is shared through the workspace."""
    from tritonformer_b200 import _lib, linear as L
    assert _lib.lib.tfb_debug_gemm_plan(m, n, k, 0) == 0
    ws = L._gemm_workspace(torch.device("cuda", 0), _lib.stream_ptr(torch.device("cuda", 0)))
    ws.zero_()
    *args, ad, bd = _operands(m, n, k, "kk")
    got = L.gemm(*args, m, n, k)
    _close(got, ad @ bd, torch.float16, k / 16)
    torch.cuda.synchronize()
    assert int(ws[8192:].count_nonzero()) > 0, "no partial tile went through the workspace"
    assert int(ws[:8192].count_nonzero()) == 0
    _check_all_epilogues(m, n, k, "kk")


def test_fewer_pair_tiles_than_pairs_run_on_the_one_wave_kernel():
    """The persistent pair kernel hands its tiles out whole, so it is left with products that fill the pairs of SMs."""
    from tritonformer_b200 import _lib
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    for tm in range(1, pairs):
        for tn in range(1, (pairs - 1) // tm + 1):
            for k in (64, 8192):
                assert _lib.lib.tfb_debug_gemm_plan(256 * tm, 256 * tn, k, tn & 1) != 0, (tm, tn, k)


@pytest.mark.parametrize("layout", ["kn", "kk", "mn", "mk"])
@pytest.mark.parametrize("m,n,k,dtype", [(3328, 1536, 136, torch.float16), (3304, 1528, 1000, torch.bfloat16)])
def test_narrow_tiles_of_the_pair_kernel(m, n, k, dtype, layout):
    """A little more than a wave of 256 x 256 tiles: 256 x 192 ones, with B in boxes of 32 columns where it is contiguous along N."""
    from tritonformer_b200 import _lib
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    wide, narrow = (-(-(-(-m // 256) * -(-n // bn)) // pairs) for bn in (256, 192))
    assert wide == narrow == 2 and _lib.lib.tfb_debug_gemm_plan(m, n, k, int(layout[1] == "n")) == 0
    _check_all_epilogues(m, n, k, layout, dtype)


@pytest.mark.parametrize("layout", ["kn", "kk", "mk"])
@pytest.mark.parametrize("m,n,k,dtype", [(3328, 1536, 136, torch.float16), (3304, 1440, 1000, torch.bfloat16), (3304, 1376, 200, torch.float16)])
def test_every_narrow_form_of_the_pair_kernel(m, n, k, dtype, layout):
    """256 x 192 tiles, whole and with one or two of the last tile's three 64-column steps outside the output."""
    from tritonformer_b200 import _lib
    assert _lib.lib.tfb_debug_gemm_pair_width(m, n, k, int(layout[0] == "m"), int(layout[1] == "n"), 1) == 192
    _check_all_epilogues(m, n, k, layout, dtype)


def test_where_the_pair_kernel_takes_narrow_tiles():
    """Not where both operands are contiguous along the output, nor where rows of B along N begin off 64-byte boundaries."""
    from tritonformer_b200 import _lib
    for k in (64, 1000, 8192):
        for a_mn, b_mn, rows_64, want in ((0, 0, 0, 192), (1, 0, 0, 192), (0, 1, 1, 192), (0, 1, 0, 256), (1, 1, 1, 256), (1, 1, 0, 256)):
            assert _lib.lib.tfb_debug_gemm_pair_width(3328, 1528, k, a_mn, b_mn, rows_64) == want
            assert _lib.lib.tfb_debug_gemm_pair_width(4096, 4608, k, a_mn, b_mn, rows_64) == 256  # four waves of wide tiles, six of narrow ones
    assert _lib.lib.tfb_debug_gemm_pair_width(512, 512, 512, 0, 0, 1) == 0  # the one-wave kernel's


@pytest.mark.parametrize("n", [1464, 1528])
def test_rows_of_b_off_64_byte_boundaries(n):
    """A little more than a wave of 256 x 256 tiles whose B, contiguous along N, keeps the wide tiles."""
    from tritonformer_b200 import _lib
    assert _lib.lib.tfb_debug_gemm_pair_width(3320, n, 200, 0, 1, 0) == 256
    for layout in ("kn", "mn"):
        _check_all_epilogues(3320, n, 200, layout)
