"""Host-side decisions that need no GPU: scratch buffers and their views, the rule that cuts decode attention's keys
over CTAs, the decode batch buckets, and the cache's serial numbers (what decode graphs are kept by)."""
import pytest
import torch

from xpu_serve_b200.cache import Cache
from xpu_serve_b200.engine.model import _bucket, _kv_bucket
from xpu_serve_b200.engine.runtime import Workspace
from xpu_serve_b200.parts.attention import decode_splits
from xpu_serve_b200.parts.base import KVNeed, StateNeed


def test_workspace_hands_out_the_same_view_until_the_buffer_grows():
    ws = Workspace(torch.device("cpu"))
    a = ws.get("x", (3, 4), torch.float32)
    assert a.shape == (3, 4) and ws.get("x", [3, 4], torch.float32) is a          # the same view again, list or tuple
    b = ws.get("x", (2, 4), torch.float32)
    assert b.data_ptr() == a.data_ptr() and b.shape == (2, 4)                      # one buffer per name and type
    assert ws.get("x", (3, 4), torch.bfloat16).data_ptr() != a.data_ptr()          # another type, another buffer
    a.fill_(7.0)
    big = ws.get("x", (10, 4), torch.float32)                                      # grows: a new buffer
    assert big.data_ptr() != a.data_ptr()
    again = ws.get("x", (3, 4), torch.float32)
    assert again is not a and again.data_ptr() == big.data_ptr(), "a view of the old buffer was handed out again"
    assert ws.get("empty", (0, 5), torch.float32).shape == (0, 5)
    ws.frozen = True
    assert ws.get("x", (10, 4), torch.float32) is big                              # fits: fine when frozen
    with pytest.raises(RuntimeError, match="frozen"):
        ws.get("x", (11, 4), torch.float32)
    with pytest.raises(RuntimeError, match="frozen"):
        ws.get("never seen", (1,), torch.float32)


def test_decode_splits_rule():
    slots = 444                                        # 148 SMs x 3 CTAs
    for tiles in (1, 8, 64, 128, 512, 4096):
        for blocks in (1, 2, 33, 64, 384, 2048):
            n = decode_splits(tiles, blocks, slots)
            assert 1 <= n <= min(blocks, 64), (tiles, blocks, n)
    assert decode_splits(8, 1, slots) == 1                                         # nothing to cut
    assert decode_splits(4096, 33, slots) == 1                                     # the tiles alone are many rounds
    assert decode_splits(64, 33, slots) == 6                                       # 8 sequences x 8 kv heads: one round of 384
    assert 8 <= decode_splits(8, 33, slots) <= 16                                  # one sequence: the combine's cost caps it
    assert decode_splits(8, 2048, slots) > 32                                      # one long sequence: fill the device
    assert decode_splits(8, 2048, slots) * 8 <= slots                              # ... in one round
    # more CTA slots never ask for fewer parts of a long sequence
    assert decode_splits(8, 2048, 2 * slots) >= decode_splits(8, 2048, slots)


def test_decode_batch_buckets():
    assert [_bucket(n) for n in (1, 5, 8, 9, 16, 17, 63, 64, 65, 96, 97)] == [1, 5, 8, 16, 16, 24, 64, 64, 96, 96, 128]
    assert all(_bucket(n) >= n for n in range(1, 300))


def test_key_length_bounds_of_decode_graphs():
    assert [_kv_bucket(n, 1 << 20) for n in (1, 1024, 1025, 1536, 1537, 2048, 2049, 3073, 100000)] == \
        [1024, 1024, 1536, 1536, 2048, 2048, 3072, 4096, 131072]
    assert all(n <= _kv_bucket(n, 1 << 20) < 2 * max(n, 1024) for n in range(1, 5000, 7))
    assert _kv_bucket(5, 300) == 300 and _kv_bucket(3100, 3500) == 3500       # never beyond the cache's limit


def test_every_cache_has_a_serial_number_of_its_own():
    def make():
        return Cache([StateNeed((2, 8)), KVNeed(2, 16, 0)], [None, None], 256, dtype=torch.float32, device="cpu")
    seen = set()
    for _ in range(5):
        c = make()
        assert c.serial not in seen
        seen.add(c.serial)
        del c                                          # the next one may get the same id(), never the same serial


def test_tokens_up_to_which_experts_take_the_product_of_few_rows():
    """16 in general, 32 where the two products have at most 1,024 CTAs of 32 weight rows."""
    from xpu_serve_b200.ops import lib
    assert lib.moe_few_tokens(16, 2 * 1024, 2048) == 16 and lib.moe_few_tokens(64, 2 * 512, 2048) == 16
    assert lib.moe_few_tokens(8, 2 * 256, 512) == 32 and lib.moe_few_tokens(16, 2 * 512, 1024) == 32
    assert lib.moe_few_tokens(16, 2 * 512, 1025) == 16 and lib.moe_few_tokens(1, 8, 8) == lib.MOE_FEW_TOKENS


class _RecordedOps:
    """Stands for the kernels: remembers which ran."""

    def __init__(self, real):
        self.real, self.ran = real, []

    def __getattr__(self, name):
        if name in ("moe_few_tokens", "MOE_FEW_TOKENS"):
            return getattr(self.real, name)
        if name.startswith("moe_max_tiles"):
            return lambda rows, experts, tile_rows=64: rows // tile_rows + min(rows, experts)
        return lambda *a, **k: self.ran.append(name)


@pytest.mark.parametrize("tokens", [1, 16, 17])
def test_experts_take_the_buffers_of_their_own_route(tokens, monkeypatch):
    """A step whose products find the experts' rows by themselves keeps no plan (each captured decode step would hold one)."""
    from types import SimpleNamespace

    from xpu_serve_b200.config.spec import RoutedExpertsSpec
    from xpu_serve_b200.parts import gated_units
    E, F, H = 64, 64, 512
    names = {"gate": "g{e}", "up": "u{e}", "down": "d{e}", "router": "r"}
    spec = RoutedExpertsSpec(hidden=H, intermediate=F, experts=E, top=2, names=names)
    weights = {"r": torch.zeros(E, H)}
    for e in range(E):
        weights.update({f"g{e}": torch.zeros(F, H), f"u{e}": torch.zeros(F, H), f"d{e}": torch.zeros(H, F)})
    ops = _RecordedOps(gated_units.ops)
    monkeypatch.setattr(gated_units, "ops", ops)
    rt = SimpleNamespace(mode="bfloat16", act_dtype=torch.bfloat16, ws=Workspace(torch.device("cpu")),
                         matrix=lambda t: t.to(torch.bfloat16), vector=lambda t: t)
    unit = gated_units.RoutedExperts(spec, weights, rt)
    assert unit.few_tokens == 16
    unit.forward(torch.zeros(tokens, H, dtype=torch.bfloat16), None)
    kept = {name for name, _ in rt.ws._bufs if name.startswith("moe_")}
    if tokens <= 16:
        assert "moe_few_rows" in ops.ran and "moe_plan" not in ops.ran
        assert kept == {"moe_logits", "moe_ids", "moe_wts", "moe_act_few", "moe_rows_few"}
    else:
        assert "moe_plan" in ops.ran and "moe_few_rows" not in ops.ran
        assert kept == {"moe_logits", "moe_ids", "moe_wts", "moe_place", "moe_source_padded", "moe_meta_padded", "moe_rows_in",
                        "moe_act", "moe_rows"}


def test_a_clamped_units_product_refuses_what_its_kernel_does_not_do(monkeypatch):
    from types import SimpleNamespace

    from xpu_serve_b200.engine import runtime
    ran = []
    fake = SimpleNamespace(gemm_small_m_ksplit=lambda *a: 1, gemm_small_m_scratch_bytes=lambda *a: 0,
                           gemm_small_m_clamped=lambda *a, **k: ran.append("clamped"), gemm_small_m=lambda *a, **k: ran.append("plain"))
    monkeypatch.setattr(runtime, "ops", fake)
    rt = runtime.Runtime.__new__(runtime.Runtime)
    rt.sm_count, rt.gemm_scratch = 148, torch.zeros(1)
    x, w, out, row = torch.zeros(2, 8), torch.zeros(16, 8), torch.zeros(2, 8), torch.zeros(16)
    clamp = (7.0, 1.702, 1.0)
    rt.few_rows_product(x, w, out, clamp=clamp)
    assert ran == ["clamped"]
    for extra in (dict(bias=row), dict(residual=out), dict(next_w=row), dict(next_x=x), dict(out_ssq=row), dict(conv={}), dict(argmax_into=row),
                  dict(swiglu=True)):
        with pytest.raises(ValueError, match="clamped"):
            rt.few_rows_product(x, w, out, clamp=clamp, **extra)
    with pytest.raises(ValueError, match="clamped"):
        rt.few_rows_product(SimpleNamespace(x=x, ssq=row, width=8, eps=1e-5, shape=x.shape), w, out, clamp=clamp)
    assert ran == ["clamped"]
    rt.few_rows_product(x, w, out, bias=row)
    assert ran == ["clamped", "plain"]


class _Places:
    """Places as a tensor on a device has them: numbers one by one, no host array of them all."""

    def __init__(self, *at):
        self.at = at

    def __len__(self):
        return len(self.at)

    def __iter__(self):
        return (torch.tensor(p) for p in self.at)

    def __array__(self, *a, **k):
        raise TypeError("can't convert a device tensor to numpy")


@pytest.mark.parametrize("many", [False, True])
def test_wanted_places_may_be_whatever_gives_numbers(many):
    from types import SimpleNamespace

    import numpy as np

    from xpu_serve_b200.engine.model import Model
    from xpu_serve_b200.engine.step import StepStager
    n = 40
    at = list(range(1, 36)) if many else [3, 7]
    kinds = [at, tuple(at), set(at), dict.fromkeys(at), np.asarray(at, dtype=np.uint8), torch.tensor(at), torch.tensor(at)[:, None], _Places(*at),
             [torch.tensor(p) for p in at], [np.int64(p) for p in at], [float(p) + 0.5 for p in at], [], np.zeros(0)]
    if many:
        kinds.append(range(1, 36))
    cache = SimpleNamespace(kv_groups=[], page_size=64, max_seq_tokens=64)
    stager = StepStager("cpu")
    ctx = stager.stage(cache, list(range(len(kinds))), [[0] * n for _ in kinds], kinds, np.zeros(len(kinds), dtype=np.int64))
    want = [i * n + p for i, k in enumerate(kinds) for p in ([] if len(k) == 0 else at)]
    assert ctx.want_rows.tolist() == want

    class Passed(Exception):
        pass

    def begin(slots, q_lens):
        raise Passed

    model = Model.__new__(Model)
    model.spec = SimpleNamespace(vocab=10)
    for places in kinds:
        with pytest.raises(Passed):                      # past the checks
            model.step(SimpleNamespace(begin_step=begin), [0], [[1] * n], [places])
    for bad in (-1, n):
        for places in ([bad] + at, np.asarray([bad] + at), {bad, *at}, _Places(bad, *at), torch.tensor([bad] + at)):
            with pytest.raises(ValueError, match="wanted place"):
                model.step(SimpleNamespace(begin_step=begin), [0], [[1] * n], [places])
