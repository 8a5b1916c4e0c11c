"""The vocabulary projection into rows without gaps (ops.lstm_project_softmax_rows)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from fractaltensor_b200 import ops as _ops
    return _ops


@pytest.mark.parametrize("T,V", [(1, 1), (37, 130), (300, 257), (100, 2000), (64, 9999), (129, 10000), (5, 49151), (9, 256)])
def test_probabilities_without_gaps(ops, T, V):
    """The same numbers as in the padded buffer, for rows that begin on a 16-byte boundary and rows that do not."""
    g = torch.Generator(device="cuda").manual_seed(V)
    P = torch.randn(64, V, device="cuda", generator=g).half()
    h = torch.randn(T, 64, device="cuda", generator=g).half()
    Pt = ops.projection_pack(P)
    rows = ops.lstm_project_softmax_rows(h, Pt, V)
    ops.check_status()
    assert rows.shape == (T, V) and (V % 128 == 0 or rows.is_contiguous())
    assert torch.equal(rows, ops.lstm_project_softmax(h, Pt, V))
    ref = torch.softmax(h.double() @ P.double(), -1)
    # fp32 logits of magnitude up to about 40: 40 * 2^-24 of them, and as much of a probability
    assert (rows.double() - ref).abs().max().item() <= 1e-5


@pytest.mark.parametrize("rows,width", [(3, 2), (40, 131), (9, 1028), (30, 5001), (5, 20001), (2, 60003), (2, 60004)])
def test_softmax_of_rows_that_begin_anywhere(ops, rows, width):
    """Rows of x, of y or of both off the 16-byte boundary; both sizes of CTA, and rows longer than the on-chip cache."""
    g = torch.Generator(device="cuda").manual_seed(width)
    x = torch.randn(rows, width, device="cuda", generator=g) * 3
    ref = torch.softmax(x.double(), -1)
    for at_x, at_y in ((0, 0), (0, 1), (3, 0), (1, 2)):
        bx, by = (torch.full((rows * width + 4,), 7.0, device="cuda") for _ in range(2))
        xs, ys = bx[at_x:at_x + rows * width].view(rows, width), by[at_y:at_y + rows * width].view(rows, width)
        xs.copy_(x)
        ops.online_softmax(xs, ys)
        # fp32 sums of up to 60004 terms and an exponential of relative error 2^-22 or so
        assert ((ys.double() - ref).abs() / ref).max().item() <= 1e-4
        assert by[:at_y].eq(7).all() and by[at_y + rows * width:].eq(7).all()


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,V,H", [(1, 8, 64), (127, 248, 128), (129, 256, 192), (257, 264, 512), (300, 2000, 640), (2500, 1000, 256), (700, 10104, 64)])
def test_product_computed_twice(ops, dt, T, V, H):
    """Probabilities without logits in memory: from the projection as it is and from its transpose, into rows without gaps and
    into padded ones, whose padding is zero.  Edges of 256 rows and columns, several row blocks a pair of CTAs."""
    from fractaltensor_b200.ops import _dtype_code, _ptr, _stream, check, lib
    g = torch.Generator(device="cuda").manual_seed(T + V)
    P = torch.randn(H, V, device="cuda", generator=g).to(dt) * 0.5
    h = torch.randn(T, H, device="cuda", generator=g).to(dt) * 0.5
    ref = torch.softmax(h.double() @ P.double(), -1)
    Pt, Vp, ws = ops.projection_pack(P), lib.ftb_projection_padded_cols(V), ops.workspace(h.device)
    scratch = torch.full((T * ((V + 255) // 256) * 16,), 255, dtype=torch.uint8, device="cuda")
    got = []
    for unpacked, ld in ((1, V), (1, Vp), (0, V), (0, Vp)):
        if lib.ftb_project_softmax_scratch_bytes(T, V, H, _dtype_code(h), unpacked) == 0:
            continue
        probs = torch.full((T, ld), 7.0, device="cuda")
        check(lib.ftb_project_softmax_fwd(_ptr(h), _ptr(P if unpacked else Pt), unpacked, _ptr(probs), ld, T, V, H, _dtype_code(h),
                                          _ptr(scratch), scratch.numel(), _ptr(ws), ws.numel(), _stream()), "ftb_project_softmax_fwd")
        ops.check_status()
        assert probs[:, V:].eq(0).all()
        got.append(probs[:, :V])
    assert len(got) >= 2 and torch.equal(ops.project_softmax_rows(h, P), got[0])
    for x in got:
        assert torch.equal(x, got[0])
        # a logit is H / 16 sums on the tensor cores, each cut off after 2^-23 of a number of up to 32 or so; a probability's
        # relative error is its logit's error, and two more of the exponential and of the row's sum
        assert ((x.double() - ref).abs() / ref.clamp_min(1e-20)).max().item() <= (H / 16 + 2) * 2.0 ** -18
        assert (x.double().sum(-1) - 1).abs().max().item() <= 2e-6


def test_packed_operand_of_many_logits(ops):
    """The transposed operand where the entry points take it: the same numbers as from the projection itself."""
    g = torch.Generator(device="cuda").manual_seed(3)
    P = torch.randn(64, 10000, device="cuda", generator=g).bfloat16()
    h = torch.randn(1700, 64, device="cuda", generator=g).bfloat16()
    a, b, c = ops.project_softmax_rows(h, P), ops.lstm_project_softmax_rows(h, ops.projection_pack(P), 10000), ops.lstm_project_softmax(h, ops.projection_pack(P), 10000)
    ops.check_status()
    assert a.is_contiguous() and torch.equal(a, b) and torch.equal(a, c)
    P4 = P[:, :9996].contiguous()  # rows of probabilities on 16 bytes, rows of the projection not
    assert (ops.project_softmax_rows(h, P4).double() - torch.softmax(h.double() @ P4.double(), -1)).abs().max().item() <= 1e-5


@pytest.mark.parametrize("T,V,twice", [(1599, 10004, False), (1600, 10004, True), (1600, 10000, True), (16002, 1002, False), (800, 20004, True)])
def test_packed_operand_around_the_rule(ops, T, V, twice):
    """16 million probabilities, rows on 16 and on 32 bytes, and rows on neither: the same within rounding on both sides."""
    from fractaltensor_b200._lib import DTYPE_F16, lib
    assert (lib.ftb_project_softmax_scratch_bytes(T, V, 128, DTYPE_F16, 0) > 0) == twice
    g = torch.Generator(device="cuda").manual_seed(T)
    P, h = torch.randn(128, V, device="cuda", generator=g).half(), torch.randn(T, 128, device="cuda", generator=g).half()
    got, padded = ops.lstm_project_softmax_rows(h, ops.projection_pack(P), V), ops.lstm_project_softmax(h, ops.projection_pack(P), V)
    ops.check_status()
    # (logits of magnitude up to about 60: 60 * 2^-24 of them, and as much of a probability)
    assert torch.equal(got, padded) and (got.double() - torch.softmax(h.double() @ P.double(), -1)).abs().max().item() <= 1e-5


def test_rows_that_are_not_finite(ops):
    """A row of logits with a NaN or +inf is NaN, the others are untouched."""
    g = torch.Generator(device="cuda").manual_seed(5)
    P, h = torch.randn(64, 512, device="cuda", generator=g).half(), torch.randn(300, 64, device="cuda", generator=g).half()
    clean = ops.project_softmax_rows(h, P)
    bad = h.clone()
    bad[7, 3], bad[290, 0] = float("nan"), float("inf")
    out = ops.project_softmax_rows(bad, P)
    ops.check_status()
    rows = torch.isnan(out).any(-1)
    assert rows[7] and rows[290] and rows.sum().item() == 2
    assert torch.equal(out[~rows], clean[~rows])


def _logits_by_value(dt, columns, T):
    """h [T,64] and P [64,V] whose product is scale(row) * (columns[0] + columns[1] + ..): in fp32 without rounding for these."""
    P = torch.zeros(64, columns[0].numel(), device="cuda", dtype=dt)
    for i, c in enumerate(columns):
        P[i] = c.to(dt)
    h = torch.zeros(T, 64, device="cuda", dtype=dt)
    h[:, :len(columns)] = 1
    h[1::3] *= 0.5
    return h, P


def _softmax_64(h, P, n):
    x = (h[:, :n, None].double() * P[None, :n].double()).sum(1)
    x = (x - x.amax(-1, keepdim=True).clamp_min(-3.4028234663852886e38))
    # (-inf and all that is far below the maximum count nothing in the sum and e^-64 as a number: the row kernel's clamp)
    return x.clamp_min(-64).exp() / x.exp().sum(-1, keepdim=True)


def _three_routes(ops, h, P):
    """The product twice, from the projection itself and from its transpose, and logits with the row kernel behind them."""
    from fractaltensor_b200.ops import _dtype_code, _ptr, _stream, check, lib
    T, (H, V) = h.shape[0], P.shape
    Pt, ws, twice, rows = ops.projection_pack(P), ops.workspace(h.device), [], torch.empty(T, lib.ftb_projection_padded_cols(V), device="cuda")
    for unpacked, ld in ((1, V), (1, rows.shape[1]), (0, V), (0, rows.shape[1])):
        n = lib.ftb_project_softmax_scratch_bytes(T, V, H, _dtype_code(h), unpacked)
        if n == 0:
            continue
        scratch, out = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty(T, ld, device="cuda")
        check(lib.ftb_project_softmax_fwd(_ptr(h), _ptr(P if unpacked else Pt), unpacked, _ptr(out), ld, T, V, H, _dtype_code(h),
                                          _ptr(scratch), n, _ptr(ws), ws.numel(), _stream()), "ftb_project_softmax_fwd")
        twice.append(out[:, :V])
    check(lib.ftb_lstm_project_softmax(_ptr(h), _ptr(Pt), _ptr(rows), T, V, H, _dtype_code(h), _ptr(ws), ws.numel(), _stream()),
          "ftb_lstm_project_softmax")
    ops.check_status()
    return twice, rows[:, :V]


def _check_against_both(got, rows, ref):
    # exponents of up to 92 in 2^-24 of themselves, 2^-22 of an exponential and of its sum: 1e-5, as for the other sizes here
    for x in got:
        assert torch.equal(torch.isinf(x), torch.isinf(rows)) and not torch.isnan(x).any()
        fin = ~torch.isinf(rows)
        assert ((x.double() - rows.double()).abs() <= 2e-5 * rows.double())[fin].all()
        assert ((x.double() - ref).abs() <= 1e-5 * ref)[fin].all() and torch.isinf(ref[~fin]).all()


@pytest.mark.parametrize("dt,value", [(torch.float16, float("-inf")), (torch.bfloat16, float("-inf")), (torch.bfloat16, -3.3895313892515355e38),
                                      (torch.bfloat16, -1e30), (torch.bfloat16, -2e9), (torch.bfloat16, 3.3895313892515355e38), (torch.bfloat16, 1e30),
                                      (torch.float16, 65504.0)])
@pytest.mark.parametrize("first,last", [(0, 1), (0, 32), (0, 128), (0, 256), (32, 64), (100, 420), (256, 512), (480, 512), (511, 512), (520, 632), (0, 632)])
def test_columns_far_from_the_others(ops, dt, value, first, last):
    """Columns of -inf (a vocabulary's padding words, masked) or of numbers at the end of the range beside ordinary ones: where a
    chunk of 32 columns, a half of 128, a tile, the short last chunk or all of the row has no other number, too."""
    g = torch.Generator(device="cuda").manual_seed(last)
    c = torch.randn(632, device="cuda", generator=g) * 4
    c[first:last] = value
    h, P = _logits_by_value(dt, [c], 300)
    twice, rows = _three_routes(ops, h, P)
    assert len(twice) == 2
    _check_against_both(twice, rows, _softmax_64(h, P, 1))


@pytest.mark.parametrize("sign", [1, -1])
def test_exponents_around_two_to_the_23(ops, sign):
    """Logits a few units apart around 2^23 / log2 e = 5814540, where a maximum's exponent stops being taken as a whole number."""
    g = torch.Generator(device="cuda").manual_seed(9)
    near = torch.randint(-40, 41, (640,), device="cuda", generator=g).float()
    near[:256] -= 80  # (a tile on one side)
    h, P = _logits_by_value(torch.bfloat16, [sign * torch.full((640,), 5799936.0, device="cuda"), sign * torch.full((640,), 14592.0, device="cuda"), near], 300)
    twice, rows = _three_routes(ops, h, P)
    # (what log2 e lacks as an fp32 number, 1.3e-8 of it, is common to a row but for the distance of its numbers)
    _check_against_both(twice, rows, _softmax_64(h, P, 3))


def test_masked_words_of_many_logits(ops):
    """The transposed operand (16 million probabilities and more) and both row strides, with the first words masked."""
    c = torch.randn(49152, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)) * 4
    c[:300] = c[40000:] = float("-inf")
    h, P = _logits_by_value(torch.bfloat16, [c], 330)
    twice, rows = _three_routes(ops, h, P)
    assert len(twice) == 4
    _check_against_both(twice, rows, _softmax_64(h, P, 1))


def test_projections_behind_one_another(ops):
    """Both passes are dependent launches: a call reads what the call before wrote, and the scratch of one is the next one's."""
    g = torch.Generator(device="cuda").manual_seed(6)
    P, h = torch.randn(512, 512, device="cuda", generator=g).half(), torch.randn(1500, 512, device="cuda", generator=g).half()

    def links(between=lambda: None):
        x = h
        for _ in range(6):
            x = ops.project_softmax_rows(x, P)
            between()
            x = (x * 400).half()
            between()
        return x

    want = links(torch.cuda.synchronize)
    for _ in range(3):
        assert torch.equal(links(), want)
    ops.check_status()


def test_sums_are_as_close_with_many_rows_as_with_few(ops):
    """A row's tiles are one pair of CTAs' when there are as many row blocks as pairs, and many pairs' when there are few rows.  The
    probabilities' sum leaves the rounding of the row's sum (the exponentials' own error is the same in both passes).  In units of
    half a rounding of a sum, 192 tiles of equal parts one behind the other come to sqrt(192 / 3) = 8, in eights to sqrt(8 / 3 +
    24 / 3) = 3.3, spread over pairs and put together by halves to about 3, with what both have within a tile and in the division.
    Measured 1.00 and 1.04 times, 2.1 and 2.2 in one running sum."""
    V, H, rows = 49152, 64, 256 * (torch.cuda.get_device_properties(0).multi_processor_count // 2 + 1)
    for dt in (torch.float16, torch.bfloat16):
        g = torch.Generator(device="cuda").manual_seed(1)
        h, P = torch.randn(rows, H, device="cuda", generator=g).to(dt), (torch.randn(H, V, device="cuda", generator=g) / 4).to(dt)
        many = ops.project_softmax_rows(h, P)
        wrong = {"many": [], "few": []}
        for first in (0, 256 * 37, rows - 512):  # (the last 256 rows' block is cut among pairs)
            few = ops.project_softmax_rows(h[first:first + 256].contiguous(), P)
            for name, p in (("many", many[first:first + 256]), ("few", few)):
                wrong[name].append(p.double().sum(-1) - 1)
            assert (few - many[first:first + 256]).abs().max().item() <= 1e-5
        ops.check_status()
        rms = {name: torch.cat(w).square().mean().sqrt().item() for name, w in wrong.items()}
        assert rms["many"] <= 1.25 * rms["few"], rms
