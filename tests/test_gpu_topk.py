"""Top-k select against torch.topk / the tie-band rule (GPU)."""
import pytest
import torch

from oracle.kascade_oracle import band_check

pytestmark = pytest.mark.gpu


def _run(scores, n_valid, k_row, k_max):
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    s = scores.to(dev).contiguous()
    rows = s.numel() // s.shape[-1]
    out = torch.full((rows, max(k_max, 1)), -7, dtype=torch.int32, device=dev)
    cnt = torch.full((rows,), -1, dtype=torch.int32, device=dev)
    nv = None if n_valid is None else n_valid.to(dev).to(torch.int32)
    kr = None if k_row is None else k_row.to(dev).to(torch.int32)
    nat.topk_select(s, nv, kr, k_max, out, cnt)
    torch.cuda.synchronize()
    return out.cpu(), cnt.cpu()


@pytest.mark.parametrize("n,k", [(4096, 300), (1000, 128), (33, 5), (4, 4), (8192, 1), (65536, 6000)])
def test_distinct_scores_exact(n, k):
    g = torch.Generator().manual_seed(n + k)
    rows = 7
    stride = (n + 3) // 4 * 4 + 8
    scores = torch.rand(rows, stride, generator=g)
    scores[:, n:] = 9.0                                   # beyond n_cols: must be ignored
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    s = scores.to(dev)
    out = torch.full((rows, k), -7, dtype=torch.int32, device=dev)
    cnt = torch.zeros(rows, dtype=torch.int32, device=dev)
    nat.topk_select(s, None, None, k, out, cnt, n_cols=n)
    torch.cuda.synchronize()
    ref = torch.topk(scores[:, :n], k, dim=-1).indices.sort(-1).values
    assert torch.equal(cnt.cpu(), torch.full((rows,), k, dtype=torch.int32))
    assert torch.equal(out.cpu().long(), ref), "index sets differ / not ascending"


def test_ties_take_lowest_index_and_negative_values():
    n = 2048
    scores = torch.zeros(3, n)
    scores[0, 100:200] = 1.0                              # 100 ones, rest zero; k = 150 -> ones + first 50 zeros
    scores[1] = -torch.arange(n, dtype=torch.float32)     # strictly decreasing, negative
    scores[2] = 0.5                                       # all tied
    out, cnt = _run(scores, None, None, 150)
    exp0 = sorted(list(range(100, 200)) + list(range(0, 50)))
    assert out[0].tolist() == exp0
    assert out[1].tolist() == list(range(150))
    assert out[2].tolist() == list(range(150))
    assert cnt.tolist() == [150, 150, 150]


def test_row_dependent_budgets_and_valid_lengths():
    g = torch.Generator().manual_seed(5)
    rows, n = 64, 2048
    scores = torch.rand(rows, n, generator=g) ** 4
    n_valid = torch.arange(rows) * 32                     # tile starts, as in an anchor prefill layer
    k_row = torch.clamp((10 * n_valid) // 100, min=128)
    out, cnt = _run(scores, n_valid, k_row, 172)
    for r in range(rows):
        want = min(int(k_row[r]), 172, int(n_valid[r]))
        assert int(cnt[r]) == want
        got = out[r, :want].tolist()
        assert got == sorted(got)
        ok, msg = band_check(scores[r], got, min(int(k_row[r]), 172), int(n_valid[r]), rel=0.0)
        assert ok, f"row {r}: {msg}"
        assert (out[r, want:] == -7).all(), "entries beyond the count must stay untouched"


def test_clustered_post_softmax_like_scores():
    # near-uniform attention: thousands of candidates within a few ulps of each other
    g = torch.Generator().manual_seed(11)
    n, k = 32768, 3244
    base = torch.full((4, n), 1.0 / n)
    scores = base * (1 + 1e-3 * torch.randn(4, n, generator=g))
    out, cnt = _run(scores, None, None, k)
    for r in range(4):
        ok, msg = band_check(scores[r], out[r].tolist(), k, n, rel=0.0)
        assert ok, msg


def test_rows_the_sample_cannot_bracket():
    """Rows on which the sampled bracket must fail, so that the histogram passes over the whole row decide: half of
    a long row tied at the threshold (the candidate lists overflow), a threshold inside a run of equal values with
    k beyond the distinct part, a step distribution, and a long row with negative values only."""
    g = torch.Generator().manual_seed(17)
    n = 40000
    rows = torch.zeros(4, n)
    rows[0] = torch.where(torch.rand(n, generator=g) < 0.5, torch.tensor(0.25), torch.rand(n, generator=g) * 0.2)
    rows[0, :100] = torch.rand(100, generator=g) + 1.0                    # 100 distinct large values, ~20000 ties at 0.25
    rows[1] = 0.125                                                        # everything tied except a few
    rows[1, 1000:1010] = 3.0
    rows[2] = (torch.arange(n) % 7).float()                                # seven plateaus
    rows[3] = -torch.rand(n, generator=g) - 1.0
    k = 5000
    out, cnt = _run(rows, None, None, k)
    assert cnt.tolist() == [k] * 4
    for r in range(4):
        vals = rows[r]
        order = torch.sort(vals, descending=True, stable=True).indices     # ties: lowest index first
        tau = vals[order[k - 1]]
        above = (vals > tau).nonzero().flatten()
        at = (vals == tau).nonzero().flatten()[: k - above.numel()]
        want = torch.cat([above, at]).sort().values
        assert torch.equal(out[r].long(), want), f"row {r}"


@pytest.mark.parametrize("n,k", [(131072, 13000), (70000, 128), (4097, 4000), (4096, 4000), (100000, 99999)])
def test_long_rows_and_extreme_budgets(n, k):
    g = torch.Generator().manual_seed(n)
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    stride = (n + 3) // 4 * 4 + 8
    scores = torch.exp(3 * torch.randn(3, stride, generator=g) - 6)        # heavy-tailed, like pooled attention mass
    scores[:, n:] = 1e9                                                    # beyond n_cols: must be ignored
    out = torch.full((3, k), -7, dtype=torch.int32, device=dev)
    cnt = torch.zeros(3, dtype=torch.int32, device=dev)
    nat.topk_select(scores.to(dev), None, None, k, out, cnt, n_cols=n)
    torch.cuda.synchronize()
    ref = torch.topk(scores[:, :n], k, dim=-1).indices.sort(-1).values
    assert cnt.tolist() == [k] * 3
    assert torch.equal(out.cpu().long(), ref)


def test_rejects_bad_arguments():
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    s = torch.zeros(2, 10, device=dev)                    # row stride not a multiple of 4
    out = torch.zeros(2, 4, dtype=torch.int32, device=dev)
    with pytest.raises(nat.KascadeNativeError):
        nat.topk_select(s, None, None, 4, out, None)


@pytest.mark.parametrize("share", [0.0, 0.05, 0.1, 0.2, 1.0])
def test_decode_budgets_inside_the_kernel_select_what_the_tensors_did(share):
    """topk_select_decode derives a row's candidates and budget from seq_lens; the general entry given them as tensors
    (computed here in 64 bits) selects the same positions.  Lengths: empty, the edges of the 128-key rule, a length whose
    share falls below the tile, one whose product with the share is a whole number, one beyond n_cols, the largest."""
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    lens = torch.tensor([0, 1, 127, 128, 129, 161, 1279, 1280, 4097, 5000, 9000, 70001], dtype=torch.int32)
    B, G, n_cols, tile = len(lens), 3, 70000, 32
    scores = torch.rand(B, G, n_cols, generator=torch.Generator().manual_seed(3)).to(dev)
    n = lens.double()
    k = torch.minimum(torch.clamp(torch.floor(share * n), min=128.0), n) - tile
    k = torch.where(n <= 128, n, k).to(torch.int32)
    k_max = 7000
    out = [torch.full((B, G, k_max), -7, dtype=torch.int32, device=dev) for _ in range(2)]
    cnt = [torch.full((B, G), -1, dtype=torch.int32, device=dev) for _ in range(2)]
    nat.topk_select(scores, lens.to(dev).view(B, 1).expand(B, G).contiguous(), k.to(dev).view(B, 1).expand(B, G).contiguous(),
                    k_max, out[0], cnt[0], n_cols=n_cols)
    nat.topk_select_decode(scores, lens.to(dev), share, tile, k_max, out[1], cnt[1], n_cols=n_cols)
    assert torch.equal(cnt[0], cnt[1]) and torch.equal(out[0], out[1])
    assert cnt[1][:, 0].tolist() == [min(int(a), int(b), n_cols, k_max) for a, b in zip(k, lens)]


def test_decode_selection_rejects_bad_arguments():
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    scores = torch.zeros(2, 2, 64, device=dev)
    out = torch.zeros(2, 2, 64, dtype=torch.int32, device=dev)
    cnt = torch.zeros(2, 2, dtype=torch.int32, device=dev)
    lens = torch.full((2,), 64, dtype=torch.int32, device=dev)
    with pytest.raises(nat.KascadeNativeError, match="share"):
        nat.topk_select_decode(scores, lens, 1.5, 32, 64, out, cnt, n_cols=64)
    with pytest.raises(nat.KascadeNativeError, match="seq_lens"):
        nat.topk_select_decode(scores, lens.long(), 0.1, 32, 64, out, cnt, n_cols=64)


@pytest.mark.parametrize("rows,n", [(1, 8191), (1, 8192), (1, 16384), (3, 32768), (8, 131071), (37, 33000), (38, 33000), (74, 16400),
                                    (75, 16400), (148, 16400), (149, 16400), (444, 700), (444, 3001), (444, 8192), (444, 8193),
                                    (444, 40001), (75, 70001), (200, 65537), (444, 65537), (444, 100003),
                                    (18, 65540), (592, 24577), (593, 24577), (741, 24577), (1183, 32772), (1184, 32772)])
@pytest.mark.parametrize("kind", ["smooth", "ties", "steps"])
def test_any_number_of_threads_selects_the_same(rows, n, kind):
    """Few long rows are split over the CTAs of a cluster (2, 4 or 8, by rows and columns), many rows get CTAs of 4 or 8
    warps each, and rows of more than 65536 scores a sample of twice the size, in clusters and out of them.  The selection
    is exact, so it equals a stable sort's, ties from the lowest index, whatever the number of CTAs: also where the
    sample's bracket fails (`ties`: half of the row has one value; `steps`: four values) and where single rows are
    short, empty or selected as a whole."""
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    g = torch.Generator().manual_seed(rows * 7 + n)
    s = torch.rand(rows, n, generator=g) ** 6
    if kind == "ties":
        s[torch.rand(rows, n, generator=g) < 0.5] = 0.125
    elif kind == "steps":
        s = torch.floor(s * 4) / 4
    stride = (n + 3) // 4 * 4
    scores = torch.nn.functional.pad(s, (0, stride - n), value=9.0).to(dev)
    n_valid = torch.full((rows,), n, dtype=torch.int32)
    k_row = torch.full((rows,), max(128, n // 10), dtype=torch.int32)
    if rows > 2:                                          # a short row, an empty one, one that is selected as a whole
        n_valid[0], n_valid[1], k_row[2] = 700, 0, n
    out = torch.full((rows, n), -7, dtype=torch.int32, device=dev)
    cnt = torch.full((rows,), -1, dtype=torch.int32, device=dev)
    nat.topk_select(scores, n_valid.to(dev), k_row.to(dev), n, out, cnt, n_cols=n)
    order = torch.sort(scores[:, :n], dim=-1, descending=True, stable=True).indices
    for r in range(rows):
        k = min(int(k_row[r]), int(n_valid[r]))
        assert int(cnt[r]) == k
        if int(n_valid[r]) == n:
            want = order[r, :k].sort().values
        else:
            m = int(n_valid[r])
            want = torch.sort(scores[r, :m], descending=True, stable=True).indices[:k].sort().values
        assert torch.equal(out[r, :k].long(), want), f"row {r}"
        assert (out[r, k:] == -7).all()


@pytest.mark.parametrize("warps,n_cols", [(8, 8193), (4, 4500)])
def test_a_cta_selects_from_one_kind_of_row_after_another(warps, n_cols):
    """More rows than the grid holds (1024 threads' worth of CTAs of 4 or 8 warps for each of 32 waves): the first CTAs take a
    second row, with the shared lists and histogram of the first.  Rows are empty, whole, tied, short or long enough to
    be sampled, in an order that puts every kind after another one."""
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    grid = nat.sm_count(0) * 1024 // warps
    rows = grid + 512
    stride = -(-n_cols // 4) * 4
    scores = torch.rand(rows, stride, generator=torch.Generator(device="cuda").manual_seed(n_cols), device=dev) ** 6
    kind = torch.arange(rows, device=dev) % 5
    scores[kind == 2] = 0.5
    n_valid = torch.tensor([0, 700, 900, 1200, n_cols], dtype=torch.int32, device=dev)[kind]
    k_row = torch.tensor([128, 700, 130, 128, n_cols // 10], dtype=torch.int32, device=dev)[kind]
    k_max = 900
    out = torch.full((rows, k_max), -7, dtype=torch.int32, device=dev)
    cnt = torch.full((rows,), -1, dtype=torch.int32, device=dev)
    nat.topk_select(scores, n_valid, k_row, k_max, out, cnt, n_cols=n_cols)
    k = torch.minimum(n_valid, k_row)
    assert torch.equal(cnt, k)
    twice = torch.cat([torch.arange(rows - grid, device=dev), torch.arange(grid, rows, device=dev)])     # a CTA's two rows
    pos = torch.arange(n_cols, device=dev)
    masked = scores[twice, :n_cols].masked_fill(pos[None, :] >= n_valid[twice, None], -1.0)
    want = torch.sort(masked, dim=-1, descending=True, stable=True).indices[:, :k_max]
    taken = torch.arange(k_max, device=dev)[None, :] < k[twice, None]
    want = torch.sort(want.masked_fill(~taken, n_cols), dim=-1).values
    assert torch.equal(out[twice].masked_fill(~taken, n_cols).long(), want)
    assert bool((out[twice][~taken] == -7).all())
