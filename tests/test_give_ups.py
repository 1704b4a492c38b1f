"""A kernel that gave up on a bounded wait: the word that it sets in host memory ends what would go on with its results.  The word is set here by the test."""
import types

import pytest
import torch

from umbrella_b200 import _lib


class Anything:
    """Takes every call and answers with itself."""

    def __call__(self, *a, **k):
        return self

    def __getattr__(self, name):
        return Anything()


@pytest.mark.parametrize("engine", ["static", "dynamic"])
def test_an_engine_looks_before_it_makes_anything_of_an_iteration(monkeypatch, engine):
    import importlib
    mod = importlib.import_module(f"umbrella_b200.speculation.{engine}_speculation_engine")
    cls = getattr(mod, f"{engine.capitalize()}SpeculationEngine")
    seen = [0]
    lib = types.SimpleNamespace(umb_give_ups_seen=lambda: seen[0], umb_error_string=lambda rc: b"an earlier kernel gave up on a wait")
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(mod, "ops", Anything())
    monkeypatch.setattr(torch.cuda, "current_stream", Anything())
    e = cls.__new__(cls)
    zeros = torch.zeros(1, 8, dtype=torch.int64)
    for name in ("parents", "depth", "depth32", "tree_bits", "tree_score", "_eos_dev", "_state", "_argmax_keys"):
        setattr(e, name, torch.zeros(8))
    e.tokens, e.position_ids, e._result, e._result_host = zeros, zeros, torch.tensor([3, 1, 5]), torch.zeros(3, dtype=torch.int64)
    e.num_nodes, e.tree_size, e._tree_pending, e.acceptance_script, e.stats = 1, 4, False, None, {"verify_calls": 0}
    e.draft_model, e.target_model = types.SimpleNamespace(kv_cache=Cache()), types.SimpleNamespace(kv_cache=Cache(), verify_forward=Anything())
    e._sample_target = Anything()
    assert e.verify() is True and (e.num_nodes, e.last_accept_length, e.target_model.kv_cache.kv_offset) == (5, 3, 4)
    seen[0], e.num_nodes = 1, 1
    with pytest.raises(RuntimeError, match="gave up"):
        e.verify()
    assert e.num_nodes == 1 and e.target_model.kv_cache.kv_offset == 4


class Cache:
    kv_offset = 0

    def gather_from_result(self, *a, **k):
        pass


@pytest.mark.gpu
@pytest.mark.parametrize("rows,awq", [(13, True), (128, True), (300, True), (13, False)])
def test_products_are_refused_from_then_on(rows, awq):
    from umbrella_b200 import ops
    K, N = 256, 256
    x = torch.zeros(rows, K, dtype=torch.float16, device="cuda:0")
    lib = _lib.load()
    ws = torch.zeros(lib.umb_awq_gemm_rows_ws_bytes(rows, K, N), dtype=torch.uint8, device="cuda:0")
    packed = torch.zeros(lib.umb_awq_packed_bytes(K, N, 128), dtype=torch.uint8, device="cuda:0")
    out = torch.empty(rows, N, dtype=torch.float16, device="cuda:0")

    def product():
        if not awq:
            return ops.gemm_f16(x, torch.zeros(N, K, dtype=torch.float16, device="cuda:0"))
        _lib.check(lib.umb_awq_gemm_rows_f16(x.data_ptr(), K, packed.data_ptr(), out.data_ptr(), N, rows, K, N, 128, None, ws.data_ptr(), ws.numel(),
                                             torch.cuda.current_stream().cuda_stream), "product")
    product()
    word = lib.umb_give_up_word()
    assert word[0] == 0
    try:
        word[0] = 1
        assert lib.umb_give_ups_seen() == 1
        with pytest.raises(RuntimeError, match="gave up"):
            product()
        with pytest.raises(RuntimeError, match="gave up"):
            _lib.raise_if_given_up()
    finally:
        word[0] = 0
    product()
    _lib.raise_if_given_up()
    torch.cuda.synchronize()
