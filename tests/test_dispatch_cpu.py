"""Which kernel a matrix product and a decode attention go to is decided on the host from sizes alone
(``Kernels._use_stream``, which is asked first up to 16 tokens, ``_route``, ``_use_pair``, ``decode_splits``). These rules were fitted to measurements at the
projection sizes of the 0.5B, 1.5B and 7B models; the test pins them for those sizes so that a change of a
threshold shows up as a decision that moved. No GPU and no library are needed: the rules read nothing but
their arguments, the object's options and its count of SMs."""
import pytest
import torch

import dataclasses

from nanoinfer_b200.config import KernelOptions
from nanoinfer_b200.csrc.lib import Kernels, _EPI

SHAPES = {      # hidden, q heads, kv heads, head dim, intermediate
    "0.5b": (896, 14, 2, 64, 4864),
    "1.5b": (1536, 12, 2, 128, 8960),
    "7b": (3584, 28, 4, 128, 18944),
}


@pytest.fixture()
def rules():
    k = Kernels.__new__(Kernels)          # the decision rules only: nothing is loaded
    k.options = KernelOptions()
    k.sm_count = 148
    return k


def projections(shape):
    hidden, heads, kv, hd, inter = SHAPES[shape]
    return {
        "qkv": ((heads + 2 * kv) * hd, hidden, _EPI["store"], True),
        "o": (hidden, heads * hd, _EPI["add"], False),
        "gate_up": (2 * inter, hidden, _EPI["swiglu"], True),
        "down": (hidden, inter, _EPI["add"], False),
    }


def test_decode_products_of_the_small_model(rules):
    """q/k/v and the output projection by the small-M kernel, gate/up and one token's down projection streamed; where the streamed
    kernel refuses its operands, gate/up goes on to the small-M kernel and the down projection to the tcgen05 one."""
    p = projections("0.5b")
    for m in (1, 8):
        assert rules._route(m, *p["qkv"]) == ("smallm", True)           # the norm folded in
        assert rules._route(m, *p["o"]) == ("smallm", False) and rules._use_stream(m, 896, 896, _EPI["add"], False) == 0
        assert rules._use_stream(m, 4864, 896, _EPI["swiglu"], True) == 1
        assert rules._use_stream(m, 896, 4864, _EPI["add"], False) == (8 if m == 1 else 0)
        assert rules._route(m, *p["gate_up"]) == ("smallm", False)      # wide output: the norm runs alone
        assert rules._route(m, *p["down"]) == ("tc", False)             # long K: split over CTAs on tcgen05
    assert rules._route(64, *p["qkv"]) == ("smallm", False)
    assert rules._route(64, *p["o"])[0] == "tc" and rules._route(64, *p["gate_up"])[0] == "tc"


def test_decode_products_of_the_large_model_go_to_tcgen05_where_the_weights_are_large(rules):
    p = projections("7b")
    assert rules._route(8, *p["qkv"])[0] == "smallm"
    assert rules._use_stream(4, 18944, 3584, _EPI["swiglu"], True) == 1 and rules._use_stream(8, 18944, 3584, _EPI["swiglu"], True) == 0
    assert rules._route(8, *p["gate_up"])[0] == "tc"
    assert rules._use_stream(1, 3584, 18944, _EPI["add"], False) == 0 and rules._route(8, *p["down"])[0] == "tc"
    lm_head = (152064, 3584, _EPI["f32"], True)
    assert rules._route(1, *lm_head) == ("tc", False)


def test_prefill_products_go_to_pairs_of_sms_when_there_are_tiles_enough(rules):
    for shape in SHAPES:
        p = projections(shape)
        rows, k, epi, _ = p["gate_up"]
        assert rules._use_pair(2048, rows, k, epi)                       # every gate/up product from 256 tokens on
        assert not rules._use_pair(64, rows, k, epi)
    rows, k, epi, _ = projections("0.5b")["o"]
    assert not rules._use_pair(2048, rows, k, epi)                       # 32 tiles of 256 x 256: the one-CTA kernel
    rows, k, epi, _ = projections("0.5b")["down"]
    assert rules._use_pair(2048, rows, k, epi)                           # the same tiles with K split in two
    for name in ("qkv", "o", "down"):
        rows, k, epi, _ = projections("7b")[name]
        assert rules._use_pair(2048, rows, k, epi)
    rules.options = dataclasses.replace(rules.options, gemm_route="tc")
    assert not rules._use_pair(2048, 9728, 896, _EPI["swiglu"])          # a forced route overrides the rule


def test_decode_attention_splits(rules):
    # TMA kernel: about 256 CTAs, at least four tiles (128 keys for heads of 64, else 64) per CTA
    assert rules.decode_splits(8, 2, 4096, 0, True, 64) == 8
    assert rules.decode_splits(1, 2, 4096, 0, True, 64) == 8
    assert rules.decode_splits(64, 2, 4096, 0, True, 64) == 2
    assert rules.decode_splits(8, 4, 4096, 0, True, 128) == 8
    assert rules.decode_splits(64, 4, 4096, 0, True, 128) == 1
    assert rules.decode_splits(8, 2, 100, 0, True, 64) == 1              # a short context is not split
    assert rules.decode_splits(8, 2, 4096, 512, True, 64) == 1           # nor is a window of 512 keys
    rules.options = dataclasses.replace(rules.options, fixed_decode_splits=5)
    assert rules.decode_splits(8, 2, 4096, 0, True, 64) == 4             # the TMA kernel's clusters: 1, 2, 4, 8, 16, 24, ...
    assert rules.decode_splits(8, 2, 4096, 0, False, 64) == 5
    rules.options = dataclasses.replace(rules.options, fixed_decode_splits=21)
    assert rules.decode_splits(8, 2, 4096, 0, True, 64) == 16


def test_decode_attention_splits_while_sms_are_idle(rules):
    # up to a cluster of eight CTAs for a context of a few tiles, as long as every CTA has an SM
    assert rules.decode_splits(1, 2, 777, 0, True, 64) == 8
    assert rules.decode_splits(1, 2, 400, 0, True, 64) == 4              # four tiles of 128 keys
    assert rules.decode_splits(24, 2, 1500, 0, True, 64) == 2
    assert rules.decode_splits(74, 2, 777, 0, True, 64) == 1             # 148 CTAs as it is
    assert rules.decode_splits(1, 2, 777, 512, True, 64) == 1            # a window: few tiles at any context
    # more than one cluster a token and kv head only where eight CTAs leave SMs idle
    assert rules.decode_splits(8, 2, 4096, 0, True, 128) == 8
    assert rules.decode_splits(1, 2, 4096, 0, True, 128) == 16


def test_decode_attention_splits_of_short_contexts(rules):
    # a replayed step plans for 256 keys at least: whatever it holds up to there is one CTA's work
    for heads_dim in (64, 128):
        for n_tokens in (1, 4, 8, 16, 37, 64):
            for keys in (17, 128, 200, 256):
                assert rules.decode_splits(n_tokens, 2, keys, 0, True, heads_dim) == 1
    # heads of 64: eight CTAs while 16 SMs are left for each token and kv head, four while 4 are (a context of four tiles: 8)
    assert [rules.decode_splits(n, 2, 512, 0, True, 64) for n in (1, 4, 8, 9, 10, 16, 32)] == [4, 4, 4, 4, 1, 1, 1]
    assert [rules.decode_splits(n, 2, 1024, 0, True, 64) for n in (1, 4, 5, 8, 16, 18, 19, 32)] == [8, 8, 4, 4, 4, 4, 2, 2]
    assert [rules.decode_splits(n, 2, 512, 0, True, 128) for n in (1, 9, 10, 18, 19, 32)] == [8, 8, 4, 4, 2, 2]


class Library:
    """A library that takes everything and notes what it was asked for."""

    def __init__(self, refuses=()):
        self.calls, self.refuses = [], refuses

    def __getattr__(self, name):
        def entry(*args):
            self.calls.append(name)
            self.args = args
            return 0 if name in self.refuses else 1 if name.endswith("_supported") else 0
        return entry

    def launches(self):
        out = [c for c in self.calls if not c.endswith("_supported")]
        self.calls.clear()
        return out


def host_side(rules, **changes):
    """``rules`` with a library that launches nothing, on tensors of the host."""
    k = rules.with_options(**changes) if changes else rules
    k._lib, k.launches, k._op_events, k._bound_stream = Library(), 0, None, 0
    k._ws_scratch = k._ws_counters = torch.zeros(1)
    return k


def operands(m, n, k, dual=False):
    return torch.zeros(m, k, dtype=torch.bfloat16), torch.zeros(2 * n if dual else n, k, dtype=torch.bfloat16), torch.zeros(m, n, dtype=torch.bfloat16)


def test_a_matrix_that_a_kernel_may_write_is_read_behind_it(rules):
    """Unless the instance was promised parameters, the products whose kernels send for W before they wait are plain launches."""
    k = host_side(rules)
    ahead = k.with_weights_ahead()
    assert ahead.weights_ahead and not k.weights_ahead and not ahead.with_options(gemm_route="tc").with_weights_ahead(False).weights_ahead
    tokens = 17
    for m, launch in ((tokens, "nib_gemm_tc_splitk"), (600, "nib_gemm_tc_pair")):
        a, w, out = operands(m, 7168, 256)
        for ops, plain in ((k, ["nib_pdl_skip_next"]), (ahead, []), (ahead.with_options(tc_splits=0), []), (ahead.with_weights_ahead(False), ["nib_pdl_skip_next"])):
            ops._gemm(a, w, None, out, m, 7168, 256, _EPI["store"])
            assert k._lib.launches() == plain + [launch]
    a, w, out = operands(12, 4096, 1024, dual=True)
    for ops, plain in ((k, ["nib_pdl_skip_next"]), (ahead, [])):
        ops._gemm(a, w, None, out, 12, 4096, 1024, _EPI["swiglu"])
        assert k._lib.launches() == plain + ["nib_gemm_stream"]


def test_the_streamed_product_is_asked_only_where_it_could_be_meant(rules, monkeypatch):
    """The host launches a prompt's step product by product: one of more than 16 tokens, or of another epilogue, costs no question."""
    k = host_side(rules)
    asked = []
    monkeypatch.setattr(Kernels, "_use_stream", lambda self, *a: asked.append(a) or 0)
    for m, epi, dual, question in ((17, "swiglu", True, False), (100, "add", False, False), (1, "store", False, False), (16, "f32", False, False), (2, "add", False, False),
                                   (16, "swiglu", True, True), (1, "add", False, True), (16, "geglu", True, True)):
        a, w, out = operands(m, 512, 256, dual)
        k._gemm(a, w, None, out, m, 512, 256, _EPI[epi])
        assert len(asked) == question, (m, epi)
        asked.clear()


@pytest.mark.parametrize("requests,late", [(12, 0), (1, 1), (3, 1)])
def test_what_comes_behind_few_tokens_of_a_prompt_is_let_in_late(rules, monkeypatch, requests, late):
    """The q/k/v product lets a decode step's attention in at once, and a prompt's only behind its weights."""
    k, m = host_side(rules), 12
    monkeypatch.setattr("nanoinfer_b200.csrc.lib._need", lambda *a, **kw: None)
    a, w, qkv = operands(m, 256, 128)
    table, pages = torch.zeros(requests, 2, dtype=torch.int32), torch.zeros(4, 1, 16, 64, dtype=torch.bfloat16)
    k.qkv_project(a, w, None, qkv, 2, 1, 64, torch.zeros(m, dtype=torch.int32), torch.zeros(m, dtype=torch.int32), None, table, 16, pages, pages, True)
    assert k._lib.launches() == ["nib_gemm_smallm_qkv"]
    assert k._lib.args[-2].value == late


def test_gated_products_of_up_to_16_tokens(rules):
    """Streamed behind a norm up to 8 tokens; with more, above the small-M product's weights, where every SM has one turn of features
    or the tcgen05 product's tiles are more than the SMs."""
    def streamed(m, hidden, inter, normed=True):
        return rules._use_stream(m, inter, hidden, _EPI["swiglu"], normed)
    for m in (1, 2, 8):
        for hidden, inter in ((64, 100), (896, 4864), (1536, 8960), (2048, 14336)):
            assert streamed(m, hidden, inter) == 1 and streamed(m, hidden, inter, False) == 0
    for m in (9, 12, 16):
        for normed in (True, False):
            for hidden, inter in ((896, 4864), (1536, 8960), (1024, 4224), (1024, 3072), (1024, 9472), (1024, 18945), (1024, 28416)):
                assert streamed(m, hidden, inter, normed) == 1, (m, hidden, inter)
            for hidden, inter in ((1024, 2816), (512, 2048), (2048, 1024), (1024, 9473), (1024, 18944), (3584, 18944), (1024, 28417)):
                assert streamed(m, hidden, inter, normed) == 0, (m, hidden, inter)
    assert streamed(17, 896, 4864) == 0 and streamed(8, 900, 4864) == 0
    assert [streamed(m, 3584, 18944) for m in (1, 6, 7, 8)] == [1, 1, 0, 0]         # several turns: the activations take the ring's room
    assert [streamed(m, 2048, 22528) for m in (12, 13, 16)] == [1, 0, 0]
    rules.options = dataclasses.replace(rules.options, gemm_route="stream")
    assert streamed(16, 512, 2048, False) == 1
    for change in (dict(gemm_route="tc"), dict(gemm_route="smallm"), dict(gemm_route=None, tc_token_tile=16), dict(gemm_route=None, smallm_cross=2)):
        rules.options = dataclasses.replace(rules.options, **change)
        assert streamed(4, 896, 4864) == 0


def test_the_down_projection_of_one_token(rules):
    """Streamed while a CTA of eight that share K holds its weights whole: one chunk of features, within a CTA's room."""
    def streamed(m, hidden, inter):
        return rules._use_stream(m, hidden, inter, _EPI["add"], False)
    for hidden, inter in ((896, 4864), (512, 8192), (1024, 4224), (1024, 5632), (1152, 5632)):
        assert streamed(1, hidden, inter) == 8 and streamed(2, hidden, inter) == 0
    for hidden, inter in ((1536, 8960), (3584, 18944), (1024, 8192), (1153, 3584), (1536, 2560), (2048, 2304), (896, 2048), (256, 16384), (896, 4900)):
        assert streamed(1, hidden, inter) == 0, (hidden, inter)
