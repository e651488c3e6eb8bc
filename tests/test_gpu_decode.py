"""Split-KV decode through the C ABI against the oracle (row L-1 of causal attention)."""
import pytest
import torch

import modern_llm_v1_b200 as m
from modern_llm_v1_b200 import inputs
from oracle import attn_oracle as ao

from gpu_util import TOL_LSE, assert_close, np32, randn_bf16, run_fwd

pytestmark = pytest.mark.gpu


def _decode(q, kc, vc, n_splits=0, want_lse=True):
    B, Hq, D = q.shape
    Hkv, L = kc.shape[1], kc.shape[2]
    o = torch.full_like(q, float("nan"))
    lse = torch.full((B, Hq), float("nan"), device=q.device) if want_lse else None
    m.flash_attn_decode(q, kc, vc, o, lse, B, L, Hq, Hkv, D, n_splits=n_splits)
    m.device_status()
    return o, lse


@pytest.mark.parametrize("B,L,Hq,Hkv,D,splits", [
    (1, 1, 1, 1, 64, 0), (2, 100, 4, 2, 64, 0), (2, 128, 6, 2, 64, 0), (2, 1000, 6, 2, 64, 0),
    (3, 777, 16, 4, 128, 0), (2, 513, 16, 1, 64, 0), (2, 300, 12, 2, 64, 0), (2, 300, 5, 1, 128, 2),
    (2, 2048, 16, 4, 64, 1), (2, 2048, 16, 4, 64, 16), (1, 700, 7, 7, 64, 3), (1, 640, 11, 1, 64, 0),
])
def test_decode_matches_oracle(B, L, Hq, Hkv, D, splits):
    q, kc, vc = randn_bf16((B, Hq, D), 1), randn_bf16((B, Hkv, L, D), 2), randn_bf16((B, Hkv, L, D), 3)
    o, lse = _decode(q, kc, vc, splits)
    wo, wl = ao.decode_c(np32(q), np32(kc), np32(vc))
    assert_close("O", o, wo)
    assert_close("LSE", lse, wl, max_abs=TOL_LSE, rel_l2=1.0)


def test_decode_config5_sampled_units():
    # B=64, cache 4096, Hq=16, Hkv=4, D=64; keys normed + RoPE'd at their true positions
    cfg = inputs.CONFIGS["c5_decode"]
    q, kc, vc, _, _ = inputs.make_decode_inputs(cfg, 20260005)
    o, lse = _decode(q.cuda(), kc.cuda(), vc.cuda())
    for b in (0, 37, 63):
        wo, wl = ao.decode_c(np32(q[b:b + 1]), np32(kc[b:b + 1]), np32(vc[b:b + 1]))
        assert_close("O", o[b:b + 1], wo)
        assert_close("LSE", lse[b:b + 1], wl, max_abs=TOL_LSE, rel_l2=1.0)


def test_decode_equals_last_row_of_the_forward_kernel():
    B, L, Hq, Hkv, D = 2, 900, 8, 2, 64
    q, k, v = randn_bf16((B, Hq, L, D), 4), randn_bf16((B, Hkv, L, D), 5), randn_bf16((B, Hkv, L, D), 6)
    o, lse = run_fwd(q, k, v)
    od, ld = _decode(q[:, :, -1].contiguous(), k, v)
    assert (od.float() - o[:, :, -1].float()).abs().max().item() <= 1e-2
    assert (ld - lse[:, :, -1]).abs().max().item() <= 1e-3


def test_decode_without_lse_and_split_invariance():
    q, kc, vc = randn_bf16((2, 8, 64), 7), randn_bf16((2, 2, 1500, 64), 8), randn_bf16((2, 2, 1500, 64), 9)
    o0, _ = _decode(q, kc, vc, 1, want_lse=False)
    for s in (2, 5, 12):
        o1, _ = _decode(q, kc, vc, s)
        assert (o0.float() - o1.float()).abs().max().item() <= 4e-3


def test_decode_is_bit_repeatable():
    # the producer re-fills a K/V stage the moment the last warp has released it: a stage that was still being read
    # would show as a run that differs from the first
    q, kc, vc = randn_bf16((16, 16, 64), 4), randn_bf16((16, 4, 3000, 64), 5), randn_bf16((16, 4, 3000, 64), 6)
    first = _decode(q, kc, vc)
    for _ in range(100):
        o, lse = _decode(q, kc, vc)
        assert torch.equal(o, first[0]) and torch.equal(lse, first[1])


@pytest.mark.parametrize("B,L,Hq,Hkv,D", [
    (1, 1025, 4, 2, 64),      # a cluster of eight over nine tiles: one CTA has two
    (1, 449, 24, 2, 128),     # a cluster, twelve heads per unit (two column tiles of the MMA)
    (120, 130, 6, 3, 64),     # more units than CTAs: ranges of whole units
    (1, 70001, 2, 1, 64),     # few long units: one unit shared by every CTA, 547 tiles
    (3, 30001, 16, 1, 128),   # sixteen heads per unit, ranges that end one unit and begin another
])
def test_every_deal_of_the_tiles_matches_the_oracle(B, L, Hq, Hkv, D):
    q, kc, vc = randn_bf16((B, Hq, D), 11), randn_bf16((B, Hkv, L, D), 12), randn_bf16((B, Hkv, L, D), 13)
    o, lse = _decode(q, kc, vc)
    o2, lse2 = _decode(q, kc, vc)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)  # whoever finishes a shared unit
    for b in sorted({0, B // 2, B - 1}):
        wo, wl = ao.decode_c(np32(q[b:b + 1]), np32(kc[b:b + 1]), np32(vc[b:b + 1]))
        assert_close("O", o[b:b + 1], wo)
        assert_close("LSE", lse[b:b + 1], wl, max_abs=TOL_LSE, rel_l2=1.0)


@pytest.mark.parametrize("B,L,Hq,Hkv,D", [(40, 3000, 6, 2, 64), (70, 1500, 8, 2, 128)])
def test_ranges_over_sequences_of_different_lengths(B, L, Hq, Hkv, D):
    # lengths from a single token to L, more than a warp's worth of sequences
    lens = torch.tensor([1 + (L - 1) * ((i * 37) % B) // (B - 1) for i in range(B)], dtype=torch.int32)
    q, kc, vc = randn_bf16((B, Hq, D), 21), randn_bf16((B, Hkv, L, D), 22), randn_bf16((B, Hkv, L, D), 23)
    cache = m.KVCache(1, B, Hq, Hkv, D, L)
    cache.k[0].copy_(kc)
    cache.v[0].copy_(vc)
    cache.set_lengths((lens - 1).tolist())
    o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq), float("nan"), device="cuda")
    cache.attend(0, q, o, lse)
    m.device_status()
    for b in (int(lens.argmin()), int(lens.argmax()), 1, 33, B - 1):
        n = int(lens[b])
        wo, wl = ao.decode_c(np32(q[b:b + 1]), np32(kc[b:b + 1, :, :n]), np32(vc[b:b + 1, :, :n]))
        assert_close(f"O[{b}]", o[b:b + 1], wo)
        assert_close(f"LSE[{b}]", lse[b:b + 1], wl, max_abs=TOL_LSE, rel_l2=1.0)


class _AbiDecode:
    """A decode through the C ABI with a workspace of its own; two units shared by every CTA, some by two."""

    def __init__(self, seed, fill=0):
        self.dims = (2, 30001, 4, 2, 64)
        B, L, Hq, Hkv, D = self.dims
        self.q, self.kc, self.vc = randn_bf16((B, Hq, D), seed), randn_bf16((B, Hkv, L, D), seed + 1), randn_bf16((B, Hkv, L, D), seed + 2)
        self.o, self.lse = torch.empty_like(self.q), torch.empty((B, Hq), device="cuda")
        self.lib = m._lib.load()
        self.ws = torch.full((self.lib.b200attn_decode_workspace_bytes(*self.dims, 0),), fill, dtype=torch.uint8, device="cuda")

    def __call__(self):
        m._lib.check(self.lib.b200attn_decode(
            *(t.data_ptr() for t in (self.q, self.kc, self.vc, self.o, self.lse)), *self.dims, 0.0, 0, self.ws.data_ptr(), self.ws.numel(),
            torch.cuda.current_stream().cuda_stream), "decode")

    def poison(self):
        self.o.fill_(float("nan"))
        self.lse.fill_(float("nan"))


def test_shared_units_do_not_depend_on_what_the_workspace_held():
    d = _AbiDecode(31)
    d()
    m.device_status()
    o, lse = d.o.clone(), d.lse.clone()
    g = torch.Generator().manual_seed(0)
    for fill in (0, 0xFF, 0x7F, 1, None, None, "its own"):
        if fill is None:
            d.ws.copy_(torch.randint(0, 256, d.ws.shape, generator=g, dtype=torch.uint8))
        elif fill != "its own":
            d.ws.fill_(fill)
        d.poison()
        d()
        m.device_status()
        assert torch.equal(d.o, o) and torch.equal(d.lse, lse), fill


def test_captured_decodes_overlap_with_other_launches():
    # Two graphs and direct launches on a third stream at the same time, each with its own workspace.  Counters taken in turn
    # from a common pool of 64 would be shared: 64 launches lie between the captures.
    ds = [_AbiDecode(41 + 3 * i) for i in range(3)]
    want = []
    for d in ds:
        d()
        m.device_status()
        want.append((d.o.clone(), d.lse.clone()))
    graphs = []
    for d in ds[:2]:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(20):
                d()
        graphs.append(g)
        for _ in range(64 - 20):
            d()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in ds]
    for _ in range(10):
        for d in ds:
            d.poison()
        torch.cuda.synchronize()
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(streams[2]):
            for _ in range(20):
                ds[2]()
        torch.cuda.synchronize()
        m.device_status()
        for d, (o, lse) in zip(ds, want):
            assert torch.equal(d.o, o) and torch.equal(d.lse, lse)
    del graphs


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("splits", [3, 5, 7, 11, 16, 40, 64])
def test_any_number_of_splits_matches_the_oracle(splits, D):
    # numbers a cluster cannot have: partial results through the workspace, added up by whoever finishes last
    B, L, Hq, Hkv = 2, 2085, 12, 2
    q, kc, vc = randn_bf16((B, Hq, D), 51), randn_bf16((B, Hkv, L, D), 52), randn_bf16((B, Hkv, L, D), 53)
    o, lse = _decode(q, kc, vc, splits)
    wo, wl = ao.decode_c(np32(q), np32(kc), np32(vc))
    assert_close("O", o, wo)
    assert_close("LSE", lse, wl, max_abs=TOL_LSE, rel_l2=1.0)
    o2, lse2 = _decode(q, kc, vc, splits)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)


@pytest.mark.parametrize("splits", [5, 12])
def test_splits_over_sequences_shorter_than_them(splits):
    # lengths of 1 .. 17 blocks: a sequence of fewer blocks than splits leaves the other CTAs without a piece
    B, L, Hq, Hkv, D = 9, 2100, 6, 2, 64
    lens = [1 + (L - 1) * b // (B - 1) for b in range(B)]
    q, kc, vc = randn_bf16((B, Hq, D), 54), randn_bf16((B, Hkv, L, D), 55), randn_bf16((B, Hkv, L, D), 56)
    lens_d = torch.tensor(lens, dtype=torch.int32, device="cuda")
    o, lse = torch.full_like(q, float("nan")), torch.full((B, Hq), float("nan"), device="cuda")
    lib = m._lib.load()
    ws = torch.empty(lib.b200attn_decode_workspace_bytes(B, L, Hq, Hkv, D, splits), dtype=torch.uint8, device="cuda")
    m._lib.check(lib.b200attn_decode_ragged(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), o.data_ptr(), lse.data_ptr(), lens_d.data_ptr(), B, L,
                                            L, Hq, Hkv, D, 0.0, splits, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "decode")
    m.device_status()
    for b, n in enumerate(lens):
        wo, wl = ao.decode_c(np32(q[b:b + 1]), np32(kc[b:b + 1, :, :n]), np32(vc[b:b + 1, :, :n]))
        assert_close(f"O[{b}]", o[b:b + 1], wo)
        assert_close(f"LSE[{b}]", lse[b:b + 1], wl, max_abs=TOL_LSE, rel_l2=1.0)
