"""The 32-bit products on the tensor cores, every operand as three bfloat16 pieces."""
import numpy as np
import pytest
import torch

from esp_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rnd(*shape, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(DEV)


def check(c, a, w, what):
    """Within rounding of the 64-bit product, element by element: every accumulation of 16 products, every addition to the running sum
    and the accumulators' sum lose at most a unit in the last place of a partial sum, together less than K / 2 of them."""
    exact = a.double() @ w.double().t()
    bound = a.shape[1] * 2.0 ** -24 * (a.double().abs() @ w.double().abs().t())
    assert torch.all((c.double() - exact).abs() <= bound), what
    return exact


@pytest.mark.parametrize("m, n, k", [
    (1, 128, 256), (15, 300, 260),     # one run of 16 rows; features and k that end inside a tile and a stage
    (16, 2048, 2048), (17, 130, 1028), (6, 6144, 2048),  # tiles shared by clusters of four, three and two CTAs, two runs of rows
    (33, 2048, 5632), (3, 640, 9300), (2, 200, 4100),   # of three; more segments than are shared; of five
    (16, 19000, 512), (64, 9600, 300),  # a CTA a tile: short tiles, several a CTA; one full run of 64 rows
    (65, 11264, 516), (200, 2304, 1100), (389, 1300, 256),   # uneven runs of rows
])
def test_dense(m, n, k):
    a, w, status = rnd(m, k), rnd(n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV)
    bias, scale = rnd(n, seed=2), rnd(m, seed=3)
    c = torch.full((m + 1, n), 7.0, device=DEV)
    ops.gemm_split(a, w, c, status, rows=m)
    assert status.item() == 0 and torch.all(c[m] == 7.0)
    exact = check(c[:m], a, w, "product")
    # no further from the 64-bit product than the chain of multiply-adds
    chain = torch.empty(m, n, device=DEV)
    ops.gemm_simt(a, w, chain)
    assert (c[:m].double() - exact).norm() <= 1.05 * (chain.double() - exact).norm()
    # bias, then scale; rows of a wider matrix; a row alone has the same bits
    wide, d = torch.zeros(m, k + 4, device=DEV), torch.empty(m, n, device=DEV)
    wide[:, :k] = a
    ops.gemm_split(wide[:, :k], w, d, status, bias=bias, row_scale=scale)
    assert torch.equal(d, (c[:m] + bias) * scale[:, None])
    one = torch.empty(1, n, device=DEV)
    for r in {0, m // 2, m - 1}:
        ops.gemm_split(a[r:r + 1], w, one, status)
        assert torch.equal(one[0], c[r]), f"row {r}"
    assert status.item() == 0


@pytest.mark.parametrize("k", [324, 1024, 1408, 2048, 4096, 5632])
@pytest.mark.parametrize("kind", ["normal", "positive", "first", "behind the middle", "last third", "several"])
def test_no_further_from_64_bits_than_the_chain_of_multiply_adds(kind, k):
    """Also where the running sum outweighs what is added to it: all of one sign, or a channel of the rows 300 times the others.  (The tensor
    core cuts its sums off, always towards zero.)  ``normal`` and ``positive`` sums lose at most a third of what the chain does from
    K = 1,024 on: a chain's error grows with the root of K, theirs is that of 128 k."""
    m, n = 64, 640
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    ours = chain = 0.0
    for seed in range(2):
        a, w = rnd(m, k, seed=2 * seed), rnd(n, k, seed=2 * seed + 1)
        if kind == "positive":
            a, w = a.abs(), w.abs()
        elif kind != "normal":
            a[:, {"first": [0], "behind the middle": [k // 2], "last third": [2 * k // 3], "several": [5, k // 4, k // 2 + 9]}[kind]] *= 300.0
        exact = a.double() @ w.double().t()
        c, d = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
        ops.gemm_split(a, w, c, status)
        ops.gemm_simt(a, w, d)
        ours += ((c.double() - exact).norm() / exact.norm()).item()
        chain += ((d.double() - exact).norm() / exact.norm()).item()
    assert status.item() == 0 and ours <= chain * (0.4 if kind in ("normal", "positive") and k >= 1024 else 1.0), (ours, chain)


def test_single_products():
    """One product an element, mantissas next to the ones whose pieces leave most behind (1.0038986 squared) among them: what is left out is at
    most 2^-25 of it, the sum of the accumulators rounds once."""
    m, n, k = 64, 3000, 64
    a, w, status = torch.zeros(m, k, device=DEV), 1 + rnd(n, k).abs().remainder(1.0), torch.zeros(1, dtype=torch.int32, device=DEV)
    w[::3] = 1.0038986 + 1e-6 * rnd(1000, k, seed=1)
    diagonal = 1 + rnd(m, seed=2).abs().remainder(1.0)
    diagonal[::2] = 1.0038986 + 1e-6 * rnd(m // 2, seed=3)
    a[torch.arange(m), torch.arange(m)] = diagonal
    c = torch.empty(m, n, device=DEV)
    ops.gemm_split(a, w, c, status)
    exact = a.double() @ w.double().t()
    assert ((c.double() - exact).abs() / exact).max() <= 1.55 * 2.0 ** -24


@pytest.mark.parametrize("counts, k", [
    ([3, 0, 66, 1, 0], 324), ([0] * 19 + [16] + [0] * 20, 324), ([1, 130, 0, 5], 324), ([64, 65, 63, 1, 200], 324), ([0, 2] * 128, 324),
    ([1] + [0] * 140 + [17, 0, 3], 324),
    ([3, 0, 66, 1], 1100), ([1, 0, 9, 0, 70], 2052), ([2, 1, 0, 1], 5632), ([0, 65, 3], 9300),      # several segments: of 512 k, of 1,024
])
def test_grouped(counts, k):
    n, rows = 300, sum(counts)
    groups = len(counts)
    offsets = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    src, w, status = rnd(50, k), rnd(groups, n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV)
    a_rows = torch.tensor(np.random.default_rng(0).integers(0, 50, rows), dtype=torch.int32, device=DEV)
    scale, c = rnd(rows, seed=2), torch.full((rows + 3, n), 7.0, device=DEV)
    ops.gemm_split(src, w, c, status, a_rows=a_rows, row_scale=scale, group_offsets=offsets, rows=rows)
    assert status.item() == 0 and torch.all(c[rows:] == 7.0)
    at, one = 0, torch.empty(1, n, device=DEV)
    for g, count in enumerate(counts):
        for r in range(at, at + count):
            if r % 9 == 0 or r == at or r == at + count - 1:
                row = a_rows[r].item()
                ops.gemm_split(src[row:row + 1], w[g], one, status)
                check(one, src[row:row + 1], w[g], f"row {r}")
                assert torch.equal(one[0] * scale[r], c[r]), f"row {r}"
        at += count


def test_infinities_nans_and_the_largest_numbers():
    """They would spread through the pieces: such elements are the chain's, the others stay as they were."""
    m, n, k = 70, 260, 512
    a, w, status = rnd(m, k), rnd(n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV)
    plain = torch.empty(m, n, device=DEV)
    ops.gemm_split(a, w, plain, status)
    a[3, 5], a[4, 7], a[66, 500] = float("inf"), float("nan"), 3.4e38
    a[5] = 0.0
    w[9, 5], w[11, 100], w[255, 3] = 0.0, -float("inf"), 3.4e38
    c, chain = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_split(a, w, c, status)
    ops.gemm_simt(a, w, chain)
    odd = torch.zeros(m, n, dtype=torch.bool, device=DEV)
    odd[[3, 4, 66]], odd[:, [11, 255]] = True, True
    odd[:, 9], odd[5] = True, True                                    # operands that changed
    assert torch.equal(c[~odd], plain[~odd])
    assert torch.equal(c.isnan(), chain.isnan()) and torch.equal(c.isinf(), chain.isinf())
    odd = ~chain.isfinite() | ~c.isfinite()
    assert torch.equal(c[odd & ~chain.isnan()], chain[odd & ~chain.isnan()])
    assert c[3, 9].isnan() and c[3, 20].isinf() and (c[5, 20] == 0).item()


@pytest.mark.parametrize("m, n, k", [(6, 40000, 2048), (6, 2048, 2048), (300, 2304, 2048)])
def test_rows_with_a_nan_take_no_longer(m, n, k):
    """One row with a NaN, then all: their elements are not made again one by one."""
    a, w, status, c = rnd(m, k), rnd(n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV), torch.empty(m, n, device=DEV)

    def milliseconds():
        times = []
        for _ in range(5):
            began, ended = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            began.record()
            for _ in range(4):
                ops.gemm_split(a, w, c, status)
            ended.record()
            torch.cuda.synchronize()
            times.append(began.elapsed_time(ended))
        return min(times)

    milliseconds()
    plain = milliseconds()
    a[m // 2, 9] = float("nan")
    assert milliseconds() < 2.5 * plain and c[m // 2].isnan().all() and c.isfinite().sum() == (m - 1) * n
    a[:, 11] = float("nan")
    assert milliseconds() < 2.5 * plain and c.isnan().all() and status.item() == 0


def test_infinities_in_every_form():
    """The chains of a shared tile, of a short one and of groups, with bias and scale behind them."""
    for m, n, k, groups in ((6, 2048, 2048, 0), (16, 19100, 512, 0), (5, 300, 1028, 3)):
        a, w, status = rnd(m, k), rnd(*([groups] if groups else []), n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV)
        a[1, 9], a[3, k - 1], a[4, 7] = float("inf"), -3.4e38, float("nan")
        bias, scale = rnd(n, seed=2), rnd(m, seed=3)
        options = {"group_offsets": torch.tensor([0, 2, 2, m], dtype=torch.int32, device=DEV)} if groups else {}
        c, chain = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
        ops.gemm_split(a, w, c, status, bias=bias, row_scale=scale, **options)
        ops.gemm_simt(a, w, chain, bias=bias, row_scale=scale, **options)
        odd = ~chain.isfinite()
        assert odd[1].all() and odd[4].all() and status.item() == 0
        assert torch.equal(c.isnan(), chain.isnan()) and torch.equal(c[odd & ~chain.isnan()], chain[odd & ~chain.isnan()])
        assert torch.equal(c[3], chain[3])


def test_refusals():
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    c = torch.zeros(4, 128, device=DEV)
    with pytest.raises(Exception, match="refused"):
        ops.gemm_split(rnd(4, 258), rnd(128, 258), c, status)          # rows that do not start on 16 bytes
    with pytest.raises(Exception, match="float32"):
        ops.gemm_split(rnd(4, 256).bfloat16(), rnd(128, 256), c, status)
    assert not ops.gemm_split_fits(rnd(4, 258), rnd(128, 258)) and ops.gemm_split_fits(rnd(4, 2048), rnd(2048, 2048))
    assert torch.all(c == 0)


@pytest.mark.parametrize("m, n, k, groups", [(6, 2048, 2048, 0), (16, 19000, 512, 0), (16, 19100, 512, 0), (200, 2304, 1100, 0), (100, 300, 2048, 30)])
def test_a_wait_that_runs_out_ends_the_kernel_in_an_orderly_way(m, n, k, groups):
    """With no polls at all every wait gives up; with few some do, and each role may be anywhere by then.  The status says so, rows behind
    the last are left alone, and the next call is right."""
    a, w, status = rnd(m, k), rnd(*([groups] if groups else []), n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV)
    options = {}
    if groups:
        options["group_offsets"] = torch.linspace(0, m, groups + 1, device=DEV).int()
    want, c = torch.empty(m, n, device=DEV), torch.full((m + 1, n), 7.0, device=DEV)
    ops.gemm_split(a, w, want, status, **options)
    assert status.item() == 0
    for polls in (0, 0, 1, 2, 3, 4, 6, 8, 16, 32, 64):
        ops.gemm_split(a, w, c, status, rows=m, polls=polls, **options)
        expired = status.item()
        assert expired == 4 if polls == 0 else expired in (0, 4)
        assert expired or torch.equal(c[:m], want)
        status.zero_()
        c[:m] = 7.0
        ops.gemm_split(a, w, c, status, rows=m, **options)
        assert status.item() == 0 and torch.equal(c[:m], want) and torch.all(c[m] == 7.0)
    with pytest.raises(Exception, match="refused"):
        ops.gemm_split(a, w, c, status, rows=m, polls=-1, **options)


@pytest.mark.parametrize("m, n, k", [(200, 2304, 1100), (16, 19100, 512), (6, 2048, 2048)])
def test_waits_do_not_count_the_kernel_before(m, n, k):
    """The product starts beside a scan of many milliseconds that lets the next kernel in at once.  Its waits get a few times the polls
    that it needs by itself."""
    a, w, status = rnd(m, k), rnd(n, k, seed=1), torch.zeros(1, dtype=torch.int32, device=DEV)
    want, c = torch.empty(m, n, device=DEV), torch.empty(m, n, device=DEV)
    ops.gemm_split(a, w, want, status)
    tokens, channels = 400_000, 32
    gates, gate = torch.zeros(tokens, 1, 2, channels, device=DEV), torch.ones(tokens, channels, device=DEV)
    out, state = torch.empty_like(gate), torch.zeros(1, channels, device=DEV)
    zeros, start, slot = torch.zeros(channels, device=DEV), torch.tensor([0, tokens], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)

    def scan():
        ops.diag_scan(gates, zeros, zeros, zeros, 8.0, gate, gate, state, start, slot, out, 1, channels, 1)

    scan()                                                            # loads its library
    torch.cuda.synchronize()
    polls = 1
    while polls < 1 << 16:
        for _ in range(3):
            ops.gemm_split(a, w, c, status, polls=polls)
        if status.item() == 0:
            break
        status.zero_()
        polls *= 2
    began, ended = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    began.record()
    scan()
    ops.gemm_split(a, w, c, status, polls=8 * polls)
    ended.record()
    assert status.item() == 0 and torch.equal(c, want), f"{polls} polls are enough for the product alone"
    assert began.elapsed_time(ended) > 2.0
