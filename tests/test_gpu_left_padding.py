"""Padded batches through the strategy (GPU): each sequence must come out exactly as if it had been run alone and
unpadded; padded query rows are zero; a padded prefill and a padded decode step launch every kernel once for the
whole batch.  The
reference ignores the mask altogether (strategies/EfficientKascadeStrategy.py:126-161), which is only right for
unpadded batches."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mask(pads, L, Lq, dtype=torch.float16, as_bool=False, right=None):
    """HF-style mask [B,1,Lq,L]: causal, the first pads[b] key positions hidden and, with `right`, also the last
    right[b] ones."""
    B = len(pads)
    qpos = torch.arange(L - Lq, L)[:, None]
    kpos = torch.arange(L)[None, :]
    ok = (kpos <= qpos)[None].repeat(B, 1, 1)
    for b, pad in enumerate(pads):
        ok[b, :, :pad] = False
        if right is not None and right[b]:
            ok[b, :, L - right[b]:] = False
    if as_bool:
        return ok[:, None].cuda()
    m = torch.zeros(B, 1, Lq, L, dtype=dtype)
    m.masked_fill_(~ok[:, None], torch.finfo(dtype).min)
    return m.cuda()


@pytest.mark.parametrize("as_bool", [False, True], ids=["additive", "bool"])
def test_left_padded_batch_equals_separate_runs(as_bool):
    from kascade_b200 import EfficientKascadeStrategy, _native as nat
    dev = torch.device("cuda")
    g = torch.Generator().manual_seed(11)
    B, H, G, D, L, layers = 3, 32, 8, 128, 416, 3
    pads = [0, 77, 160]
    hm = [list(range(G)), [3, 3, 0, 7, 1, 6, 2, 5], list(range(G))]

    def make():
        return EfficientKascadeStrategy([0, 2], "x/y", k=25, tile_size=32, rolling_prefill=True, head_mapping=hm,
                                        register=False)

    class M:
        num_key_value_groups = H // G

    qs = [(torch.randn(B, H, L + 1, D, generator=g) / D ** 0.5).half().to(dev) for _ in range(layers)]
    ks = [torch.randn(B, G, L + 1, D, generator=g).half().to(dev) for _ in range(layers)]
    vs = [torch.randn(B, G, L + 1, D, generator=g).half().to(dev) for _ in range(layers)]
    batch = make()
    alone = [make() for _ in range(B)]
    mask_p = _mask(pads, L, L, as_bool=as_bool)
    mask_d = _mask(pads, L + 1, 1, as_bool=as_bool)
    for phase in ("prefill", "decode"):
        for l in range(layers):
            m = M()
            m.layer_idx = l
            if phase == "prefill":
                q, k, v, mask = qs[l][:, :, :L], ks[l][:, :, :L], vs[l][:, :, :L], mask_p
            else:
                q, k, v, mask = qs[l][:, :, L:], ks[l], vs[l], mask_d
            n0 = nat.launch_count
            got, _ = batch.attention_forward(m, q, k, v, mask, D ** -0.5)
            if phase == "prefill":                       # one launch per kernel kind for the whole padded batch
                assert nat.launch_count - n0 == {0: 4, 1: 1, 2: 5}[l], f"layer {l}: {nat.launch_count - n0} launches"
            else:                                        # and so does a padded decode step (no loop over sequences)
                assert nat.launch_count - n0 == {0: 3, 1: 1, 2: 4}[l], f"decode layer {l}: {nat.launch_count - n0} launches"
            for b, pad in enumerate(pads):
                qb = q[b:b + 1, :, pad:] if phase == "prefill" else q[b:b + 1]
                want, _ = alone[b].attention_forward(m, qb, k[b:b + 1, :, pad:], v[b:b + 1, :, pad:], None, D ** -0.5)
                if phase == "prefill":
                    assert torch.equal(got[b:b + 1, pad:], want), f"{phase} layer {l} sequence {b}"
                    assert bool((got[b, :pad] == 0).all()), "padded query rows must be zero"
                else:
                    assert torch.equal(got[b:b + 1], want), f"{phase} layer {l} sequence {b}"
    assert nat.read_status() == 0


def test_right_and_mixed_padding_equal_separate_runs():
    """Right padding (sequence at the start of its slot), left padding and a mix, lengths that are not multiples
    of the tile, one sequence of only 150 tokens: the prefill of the whole batch in one launch per kernel
    equals the separate unpadded runs bit for bit."""
    from kascade_b200 import EfficientKascadeStrategy, _native as nat
    dev = torch.device("cuda")
    g = torch.Generator().manual_seed(12)
    B, H, G, D, L, layers = 4, 32, 8, 128, 400, 3
    left, right = [0, 0, 50, 0], [0, 123, 31, 250]
    hm = [list(range(G)), [1, 0, 0, 7, 4, 6, 2, 5], list(range(G))]

    def make():
        return EfficientKascadeStrategy([0, 2], "x/y", k=30, tile_size=32, rolling_prefill=True, head_mapping=hm,
                                        register=False)

    class M:
        num_key_value_groups = H // G

    batch, alone = make(), [make() for _ in range(B)]
    mask = _mask(left, L, L, right=right)
    for l in range(layers):
        q = (torch.randn(B, H, L, D, generator=g) / D ** 0.5).half().to(dev)
        k = torch.randn(B, G, L, D, generator=g).half().to(dev)
        v = torch.randn(B, G, L, D, generator=g).half().to(dev)
        m = M()
        m.layer_idx = l
        got, _ = batch.attention_forward(m, q, k, v, mask, D ** -0.5)
        for b in range(B):
            lo, hi = left[b], L - right[b]
            want, _ = alone[b].attention_forward(m, q[b:b + 1, :, lo:hi], k[b:b + 1, :, lo:hi], v[b:b + 1, :, lo:hi], None,
                                                 D ** -0.5)
            assert torch.equal(got[b:b + 1, lo:hi], want), f"layer {l} sequence {b}"
            assert bool((got[b, :lo] == 0).all()) and bool((got[b, hi:] == 0).all()), "rows outside a sequence must be zero"
    assert nat.read_status() == 0


def test_unpadded_mask_takes_the_batched_path():
    from kascade_b200 import EfficientKascadeStrategy
    s = EfficientKascadeStrategy([0], "x/y", k=10, tile_size=32, head_mapping=[list(range(8))] * 2, register=False)
    assert s._padding(_mask([0, 0], 64, 64), 2, 64) is None
    assert s._padding(None, 2, 64) is None
    assert s._padding(_mask([0, 5], 64, 64), 2, 64) == ([0, 5], [64, 59])
    assert s._padding(_mask([0, 5], 64, 64, right=[10, 0]), 2, 64) == ([0, 5], [54, 59])


@pytest.mark.parametrize("L", [1, 8, 9, 64, 129])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_zero_padding_clears_exactly_the_rows_outside(L, dtype):
    """Sequences that fill their slot, are empty, start or end inside a group of rows, or are given without first rows."""
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    starts = [0, 0, min(3, L - 1), L - 1, L // 2]
    lens = [L, 0, max(L - 3 - (L > 8), 0), 1, L - L // 2]
    for first in (starts, None):
        out = torch.full((len(lens), L, 5, 8), 7.0, dtype=dtype, device=dev)
        rg = (None if first is None else torch.tensor(first, dtype=torch.int32, device=dev),
              torch.tensor(lens, dtype=torch.int32, device=dev))
        nat.zero_padding(out, nat.ragged(*rg))
        pos = torch.arange(L)
        for b, n in enumerate(lens):
            s = 0 if first is None else first[b]
            inside = (pos >= s) & (pos < s + n)
            assert bool((out[b].cpu()[inside] == 7).all()) and bool((out[b].cpu()[~inside] == 0).all()), (L, b)


def _small_strategy():
    from kascade_b200 import EfficientKascadeStrategy
    return EfficientKascadeStrategy([0], "x/y", k=20, tile_size=32, head_mapping=[[0, 1], [1, 0]], register=False)


def _layer(index):
    class M:
        num_key_value_groups = 4
        layer_idx = index
    return M()


@pytest.mark.filterwarnings("ignore:The CUDA Graph is empty")
def test_a_padded_prompt_is_refused_under_capture():
    """A padded prompt's rows and lengths are copied from the host, so a graph would hold the addresses of tensors that the
    next mask replaces: capturing it is refused, also when the mask has been seen before, and the strategy stays usable."""
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    g = torch.Generator(device="cuda").manual_seed(2)
    B, H, G, D, L = 2, 8, 2, 128, 200
    q = torch.randn(B, H, L, D, generator=g, device=dev).half()
    k, v = (torch.randn(B, G, L, D, generator=g, device=dev).half() for _ in range(2))
    s, mask = _small_strategy(), _mask([0, 37], L, L)
    want = [s.attention_forward(_layer(l), q, k, v, mask, D ** -0.5)[0] for l in range(2)]
    torch.cuda.synchronize()
    for l in range(2):
        with pytest.raises(nat.KascadeNativeError, match="capture"):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                s.attention_forward(_layer(l), q, k, v, mask, D ** -0.5)
    for l in range(2):
        assert torch.equal(s.attention_forward(_layer(l), q, k, v, mask, D ** -0.5)[0], want[l])


def test_zero_padding_of_more_sequences_than_a_grid_row_holds():
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    B, L = 65537, 3
    lens = torch.arange(B, dtype=torch.int32, device=dev) % (L + 1)
    out = torch.ones(B, L, 8, dtype=torch.float16, device=dev)
    nat.zero_padding(out, nat.ragged(None, lens))
    inside = torch.arange(L, device=dev)[None, :] < lens[:, None]
    assert torch.equal(out, inside[:, :, None].expand(B, L, 8).half())


def test_the_clear_of_a_padded_layer_is_tallied():
    """Every kernel of a padded prompt's layer is in a tally: the computing ones in launch_count, the clear of the padding in
    clear_count; an unpadded layer and an empty output clear nothing."""
    from kascade_b200 import _native as nat
    dev = torch.device("cuda")
    B, H, G, D, L = 2, 8, 2, 128, 200
    q = torch.zeros(B, H, L, D, dtype=torch.float16, device=dev)
    k = torch.zeros(B, G, L, D, dtype=torch.float16, device=dev)
    s = _small_strategy()
    for mask, clears in ((_mask([0, 37], L, L), 1), (None, 0)):
        for l, launches in ((0, 4), (1, 1)):
            before = nat.launch_count, nat.clear_count
            s.attention_forward(_layer(l), q, k, k, mask, 1.0)
            assert (nat.launch_count - before[0], nat.clear_count - before[1]) == (launches, clears), (l, clears)
    before = nat.clear_count
    nat.zero_padding(q.new_empty(0, L, D), nat.ragged(None, torch.zeros(1, dtype=torch.int32, device=dev)))
    assert nat.clear_count == before


def test_one_strategy_sees_a_second_mask_and_an_edited_one():
    """Rows and lengths are copied to the device once per mask: another mask, and the same one edited in place, replace them."""
    dev = torch.device("cuda")
    g = torch.Generator(device="cuda").manual_seed(3)
    B, H, G, D, L = 3, 8, 2, 128, 300
    q = torch.randn(B, H, L, D, generator=g, device=dev).half()
    k, v = (torch.randn(B, G, L, D, generator=g, device=dev).half() for _ in range(2))
    s = _small_strategy()
    first, second = _mask([0, 40, 90], L, L), _mask([33, 0, 5], L, L, right=[0, 9, 0])
    for turn, mask in enumerate([first, second, second, first]):
        if turn == 2:
            mask.copy_(_mask([150, 1, 0], L, L))
        alone = _small_strategy()
        for l in range(2):
            got = s.attention_forward(_layer(l), q, k, v, mask, D ** -0.5)[0]
            want = alone.attention_forward(_layer(l), q, k, v, mask.clone(), D ** -0.5)[0]
            assert torch.equal(got, want), f"mask {turn}, layer {l}"
