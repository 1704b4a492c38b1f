"""What the tensor-level calls and the model do around the native library, on the CPU with a library that only records."""
import ctypes as C

import pytest
import torch

from umbrella_b200 import _lib_seq as S
from umbrella_b200 import ops_seq as K


class Recorder:
    """Every entry point returns 0 and writes nothing."""

    def __getattr__(self, name):
        return lambda *a: 0


@pytest.fixture
def recorder(monkeypatch):
    lib = Recorder()
    monkeypatch.setattr(S, "load", lambda *a, **k: lib)
    monkeypatch.setattr(K, "_stream", lambda: 0)
    monkeypatch.setattr(K, "_mode", lambda t: S.UMBS_BF16)
    dirty = lambda *a, **k: torch.full(a[0], 7.0, **k)               # memory that something else has used
    monkeypatch.setattr(K.torch, "empty", dirty)
    return lib


@pytest.mark.parametrize("max_rows,cleared", [(None, False), (6, False), (5, True), (0, True)])
def test_rows_that_a_product_is_told_to_leave_out_are_zero(recorder, max_rows, cleared):
    a, w = torch.ones(6, 8, dtype=torch.bfloat16), torch.ones(4, 8, dtype=torch.bfloat16)
    out = K.gemm(a, w, max_rows=max_rows)
    assert bool((out == 0).all()) == cleared
    assert K.gemm(a, w, rows=3, max_rows=2).eq(0).all()              # of the rows asked for, not of a's


# ---------------------------------------------------------------------------------------------- a kernel that gave up
def test_a_give_up_is_raised_before_anything_is_made_of_the_results(monkeypatch):
    """The library reports it as a word that needs no synchronisation; the model looks before a step, the engine behind the copy
    of the sampled tokens."""
    from umbrella_b200.models import seq_model
    from umbrella_b200.speculation import batch_engine
    seen = [0]
    monkeypatch.setattr(S, "load", lambda *a, **k: type("Lib", (), {"umbs_give_ups_seen": staticmethod(lambda: seen[0])})())
    model = seq_model.SeqStateModel.__new__(seq_model.SeqStateModel)
    model.spec = seq_model.SeqModelSpec(width=8, vocab=5, layers=[])
    model.cache, model.device, model.max_length = None, torch.device("cpu"), None
    assert model.forward([]).shape == (0, 5)
    engine = batch_engine.BatchDecodingEngine.__new__(batch_engine.BatchDecodingEngine)
    engine.model = model
    engine.sample = lambda logits: logits.argmax(-1)
    assert engine._take(torch.eye(3)) == [0, 1, 2]
    seen[0] = 1
    with pytest.raises(RuntimeError, match="gave up"):
        engine._take(torch.eye(3))
    with pytest.raises(RuntimeError, match="gave up"):
        model.forward([])
    with pytest.raises(RuntimeError, match="gave up"):
        S.check(-5, "forward")


# ---------------------------------------------------------------------------------------------- what the library refuses
@pytest.mark.skipif(torch.cuda.is_available(), reason="memory of the host: only where no kernel could follow")
@pytest.mark.parametrize("tokens", [1, 40, 128])
@pytest.mark.parametrize("dtype", [-1, 2, 7])
def test_retention_refuses_types_that_it_does_not_have(tokens, dtype):
    """Before anything is launched, whichever kernels the step's length would take."""
    heads, dim, vdim = 1, 8, 8
    batch = S.Batch()
    batch.n_tokens, batch.n_seqs, batch.max_seq_len = tokens, 1, tokens
    keep = [torch.zeros(tokens * 64) for _ in range(6)]
    p = [t.data_ptr() for t in keep]
    got = S.load().umbs_retention_ex(dtype, p[0], 2 * heads * (dim + vdim), C.byref(batch), heads, dim, vdim, 0, None, p[1], 1e-6, p[2], p[3], None, p[4],
                                     tokens * 256, None, p[5], None)
    assert got == -1                                                 # UMB_ERR_ARG


# ---------------------------------------------------------------------------------------------- kernels that follow one another
def test_tensor_memory_is_taken_before_the_next_kernel_is_let_in():
    """A product of the next launch takes its tensor memory ahead of its wait: beside a block that has let it in and has none itself, neither
    would ever go on.  So in every kernel the allocation stands in front of what lets the next one in."""
    import glob
    import os
    import re
    seen = 0
    for path in glob.glob(os.path.join(os.path.dirname(S.__file__), "csrc", "seq", "*.cu")):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for body in text.split("__global__")[1:]:
            body = body[:re.search(r"^}", body, re.M).end()]
            alloc = re.search(r"tmem_alloc\(|tcgen05\.alloc", body)
            let_in = re.search(r"chain_wait\(\)|chain_next\(\)", body)
            if alloc and let_in:
                seen += 1
                assert alloc.start() < let_in.start(), (path, body[:120])
            if alloc and "chain_wait_only()" in body:
                assert let_in, path
    assert seen >= 5


def test_the_native_calls_load_in_a_process_without_torch():
    """A build check imports the package and nothing else."""
    import subprocess
    import sys
    code = "import sys; from umbrella_b200 import _lib_seq; assert 'torch' not in sys.modules; assert _lib_seq.load_calls() is not _lib_seq.DECLINES"
    subprocess.run([sys.executable, "-c", code], check=True, cwd=S.__file__.rsplit("/", 2)[0])


def test_the_native_calls_are_found_for_what_they_were_made_with(monkeypatch):
    """Sources, torch and Python: the module holds layouts of all three, and a file made for others must not be loaded."""
    import os
    import sysconfig

    from umbrella_b200 import build
    here = build.calls_path()
    assert build.calls_path() == here and build.build_calls() == here and os.path.exists(here)
    paths = {here}
    with monkeypatch.context() as m:
        m.setattr(torch, "__version__", "2.99.0")
        paths.add(build.calls_path())
    with monkeypatch.context() as m:
        m.setattr(sysconfig, "get_config_var", lambda name: "cpython-399")
        paths.add(build.calls_path())
    with monkeypatch.context() as m:
        m.setattr(build, "_CALLS_DEPS", build._CALLS_DEPS[:1] + [__file__])
        paths.add(build.calls_path())
    assert len(paths) == 4 and sum(map(os.path.exists, paths)) == 1


@pytest.mark.parametrize("what", ["no compiler", "a build that fails", "a file that does not load"])
def test_calls_do_without_the_native_way(monkeypatch, recorder, tmp_path, what):
    """Whatever keeps the module from being had is said once, and the wrappers' own way goes on."""
    from umbrella_b200 import build
    monkeypatch.setattr(S, "calls", None)
    if what == "a file that does not load":
        (tmp_path / "x.so").write_bytes(b"not a library")
        monkeypatch.setattr(build, "build_calls", lambda *a, **k: str(tmp_path / "x.so"))
    else:
        monkeypatch.setattr(build, "calls_path", lambda: str(tmp_path / "none.so"))
        monkeypatch.setattr(build.shutil, "which", lambda name: str(tmp_path / "g++") if what == "no compiler" else "/bin/false")
        monkeypatch.setattr(build, "_nvcc", lambda: "/usr/local/cuda/bin/nvcc")
    with pytest.warns(RuntimeWarning, match="ctypes"):
        assert S.load_calls() is S.DECLINES
    assert S.load_calls() is S.DECLINES and S.DECLINES.gemm(1, 2) is None
    a, w = torch.ones(6, 8, dtype=torch.bfloat16), torch.ones(4, 8, dtype=torch.bfloat16)
    assert K.gemm(a, w).shape == (6, 4)


def test_threads_at_their_first_call_build_once(monkeypatch, recorder, tmp_path):
    """Two builds at a time would write and move the same temporary file."""
    import threading
    import time

    from umbrella_b200 import build
    made = []

    def slow(*a, **k):
        made.append(threading.get_ident())
        time.sleep(0.2)
        raise RuntimeError("not here")
    monkeypatch.setattr(build, "build_calls", slow)
    monkeypatch.setattr(S, "calls", None)
    got = []
    with pytest.warns(RuntimeWarning, match="not here"):
        threads = [threading.Thread(target=lambda: got.append(S.load_calls())) for _ in range(4)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert got == [S.DECLINES] * 4 and len(made) == 1
