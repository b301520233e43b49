"""The short way into the library (host_binding.cpp) against the general one (ctypes): the same results bit for bit over the forms
that it accepts, and whatever else it is handed goes the general way, with that way's results and errors."""
import sys
import threading
import time

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from litetopk_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SC = synth.REFCOMPAT_SCALE


@pytest.fixture
def both(monkeypatch):
    """f -> (result of f by the short way, by the general one), and whether the short way took it."""
    host = _lib.host()
    assert host is not None, "the module of host_binding.cpp is missing"

    def run(f):
        took = []

        class Spy:
            def __getattr__(self, name):
                def call(*args):
                    took.append(getattr(host, name)(*args))
                    return took[-1]
                return call
        monkeypatch.setattr(_lib, "_host", Spy())
        short = f()
        monkeypatch.setattr(_lib, "_host", None)
        general = f()
        torch.cuda.synchronize()
        return short, general, [r is not None for r in took]
    return run


def _same(a, b):
    a, b = (x if isinstance(x, (tuple, list)) else (x,) for x in (a, b))
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert x.shape == y.shape and x.dtype == y.dtype and x.stride() == y.stride() and torch.equal(x, y)


def _prefill(T, h, k, S, q_type, cache):
    w = synth.Workload("t", tokens=T, heads=h, topk=k, s_kv=S, overlap=(0.7, 0.7))
    idx = synth.make_topk(w, seed=5).to(DEV)
    rows = synth.make_kv_cache(S, seed=5, device=DEV, mode="native" if cache == "native" else "refcompat")
    kv = api.prepare_kv(rows) if cache == "native" else api.prepare_kv(rows, SC)
    x = torch.randn((T, h, 576), generator=torch.Generator().manual_seed(5)).to(DEV)
    q = x.to(torch.bfloat16) if q_type == "bf16" else synth.e4m3_codes(x / SC)
    return q, kv, idx, ({} if cache == "native" else dict(kv_scale=SC, q_scale=SC))


@pytest.mark.parametrize("T,h,k,S,q_type,cache", [
    (2, 64, 256, 2048, "bf16", "fp8"), (2, 64, 1024, 4096, "e4m3", "fp8"), (16, 8, 128, 999, "e4m3", "fp8"), (1, 128, 256, 777, "bf16", "fp8"),
    (6, 64, 512, 3001, "bf16", "native"), (200, 64, 256, 2048, "bf16", "fp8"), (8, 32, 32, 640, "e4m3", "fp8")])
def test_sparse_prefill(both, T, h, k, S, q_type, cache):
    q, kv, idx, scales = _prefill(T, h, k, S, q_type, cache)
    for q_, kv_, extra in ((q, kv, {}), (q if q_type == "bf16" else q.view(torch.float8_e4m3fn), kv, dict(seq_space=S + 1, job_tokens=T + 4 * 128 // h)),
                           (q, torch.cat([kv, kv], dim=1)[:, :576], {})):                    # rows of a wider pitch
        short, general, took = both(lambda: api.sparse_prefill(q_, kv_, idx, synth.SM_SCALE, **scales, **extra))
        assert took == [True]
        _same(short, general)


def test_what_is_not_plain_goes_the_general_way(both):
    q, kv, idx, scales = _prefill(4, 64, 256, 2048, "bf16", "fp8")
    call = lambda q=q, kv=kv, idx=idx, **kw: api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **{**scales, **kw})      # noqa: E731
    plain = call()
    wide = torch.cat([q, q], dim=2)[:, :, :576]
    for f in (lambda: call(q=wide), lambda: call(idx=torch.cat([idx, idx], dim=1)[:, :256]), lambda: call(kv=kv[:, None]),
              lambda: call(kv_scale=torch.tensor(SC))):
        short, general, took = both(f)
        assert took == [False]
        _same(short, general)
        _same(short, plain)
    short, general, took = both(lambda: call(out=torch.empty_like(plain[0])))
    assert took == []
    _same(short, plain)
    short, general, took = both(lambda: call(q_scale=None))                                  # derived with a synchronisation
    assert took == [False]
    _same(short, general)
    for kw, exc in ((dict(q=q[:, :48]), ValueError), (dict(q=q.float()), TypeError), (dict(idx=idx.long()), TypeError),
                    (dict(idx=idx[:2]), ValueError), (dict(kv=kv[:, :512]), ValueError), (dict(q=q.cpu()), ValueError),
                    (dict(job_tokens=2), ValueError), (dict(q=None), TypeError)):
        for way in (_lib.host(), None):
            with pytest.MonkeyPatch.context() as m:
                m.setattr(_lib, "_host", way)
                with pytest.raises((exc, AttributeError) if kw.get("q", 0) is None else exc):
                    call(**kw)
    for way in (_lib.host(), None):                                                          # refused by the library
        with pytest.MonkeyPatch.context() as m:
            m.setattr(_lib, "_host", way)
            with pytest.raises(_lib.LiteDSAError) as e:
                call(idx=idx[:, :254].contiguous())
            assert e.value.code == _lib.ERR_SHAPE
            with pytest.raises(_lib.LiteDSAError) as e:
                call(q_scale=0.0)
            assert e.value.code == _lib.ERR_SHAPE


@pytest.mark.parametrize("T,h,S,n_comp,sink", [(2, 64, 300, 0, False), (24, 16, 77777, 607, True), (4, 32, 5000, 39, True)])
def test_dsv4_ranges(both, T, h, S, n_comp, sink):
    g = torch.Generator(device=DEV).manual_seed(6)
    q, kr = (torch.empty(s, dtype=torch.bfloat16, device=DEV).normal_(generator=g) for s in ((T, h, 576), (S, 576)))
    kc = torch.empty((n_comp, 576), dtype=torch.bfloat16, device=DEV).normal_(generator=g) if n_comp else None
    sk = torch.randn((h,), generator=g, device=DEV) if sink else None
    short, general, took = both(lambda: api.dsv4_c128a_bf16(q, kc, kr, S - T, synth.SM_SCALE, attn_sink=sk))
    assert took == [True]
    _same(short, general)
    short, general, took = both(lambda: api.dsv4_c128a_bf16(q, q.new_empty((0, 576)), kr, S - T, synth.SM_SCALE, heads=h))
    assert took == []
    _same(short, general)


@pytest.mark.parametrize("dims", [2, 3])
def test_dsv4_lists(both, dims):
    T, h, S = 8, 32, 3000
    g = torch.Generator(device=DEV).manual_seed(7)
    q, kc, kr = (torch.empty(s, dtype=torch.bfloat16, device=DEV).normal_(generator=g) for s in ((T, h, 512), (S // 128, 512), (S, 512)))
    q, kv, idx, pref, lo, hi, counts = synth.dsv4_rank_space_operands(q, kc, kr, S - T, h, 128, 128)
    kv, idx = (x.reshape(x.shape[0], -1) if dims == 2 else x.reshape(x.shape[0], 1, -1) for x in (kv, idx))
    sink = torch.randn((128,), generator=g, device=DEV)

    def call(in_place=False):
        out, lse = torch.empty((T * h // 128, 128, 512), dtype=torch.bfloat16, device=DEV), torch.empty((T * h // 128, 128), device=DEV)
        api.dsv4_masked_mla_bf16_out(q, kv, idx, pref, lo, hi, counts, synth.SM_SCALE, h, out, lse, sink)
        return out, lse
    short, general, took = both(call)
    assert took == [True]
    _same(short, general)


@pytest.mark.parametrize("T,Hi,S,k,scale", [(3, 32, 1001, 64, True), (36, 64, 5000, 1024, True), (2, 128, 4096, 512, False)])
def test_lite_topk(both, T, Hi, S, k, scale):
    q, kk, w, ks = (x.to(DEV) for x in synth.make_indexer_operands(T, S, Hi, seed=8))
    short, general, took = both(lambda: api.lite_topk(q, kk, w, ks if scale else None, k, S - T))
    assert took == [True]
    _same(short, general)
    short, general, took = both(lambda: api.lite_topk(q, kk, w, ks, k, S - T, logits_workspace=torch.empty((T, S + 5), device=DEV)))
    assert took == []
    assert torch.equal(short.sort(dim=1).values, general.sort(dim=1).values)


@pytest.mark.filterwarnings("ignore:Warning only once for all operators")      # that kernels are overridden
def test_exceptions_below_are_those_of_the_general_way():
    q, kv, idx, scales = _prefill(2, 64, 256, 2048, "e4m3", "fp8")
    xi = [x.to(DEV) for x in synth.make_indexer_operands(8, 1024, 32, seed=8)]
    r = torch.randn((24, 16, 576), device=DEV).to(torch.bfloat16)
    calls = (lambda: api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales), lambda: api.lite_topk(*xi, 64, 1016),
             lambda: api.dsv4_c128a_bf16(r, None, r[:, 0], 0, synth.SM_SCALE))

    class Own(Exception):
        pass

    def refuse(*args, **kwargs):
        raise Own("from below")
    for way in (_lib.host(), None):
        with pytest.MonkeyPatch.context() as m:
            m.setattr(_lib, "_host", way)
            for f in calls:
                f()
                lib = torch.library.Library("aten", "IMPL")      # noqa: TOR901
                try:
                    for op in ("empty.memory_format", "empty_strided"):
                        lib.impl(op, refuse, "CUDA")
                    with pytest.raises(Own, match="from below"):
                        f()
                finally:
                    lib._destroy()
            torch.cuda.synchronize()
            torch.cuda.set_per_process_memory_fraction(1e-6)
            try:
                with pytest.raises(torch.OutOfMemoryError):      # 64 GB of positions
                    api.lite_topk(*xi, 2 ** 31 - 1, 1016)
            finally:
                torch.cuda.set_per_process_memory_fraction(1.0)
            calls[0]()


@pytest.mark.parametrize("T,h,k", [(592, 64, 64), (594, 64, 64), (594, 64, 128), (296, 128, 512), (297, 128, 512), (297, 128, 640)])
def test_bf16_queries_with_a_pass_of_their_own_go_the_general_way(both, T, h, k):
    """The line between both ways (296 tiles, lists of 512 entries or unions of 128) is drawn in both."""
    q, kv, idx, scales = _prefill(T, h, k, 2048, "bf16", "fp8")
    short, general, took = both(lambda: api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales))
    assert took == [not api._quantise_first(T * h // 128, 128 // h, 128 // h * k)]
    _same(short, general)


class _Count(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.n = getattr(self, "n", 0) + 1
        return func(*args, **(kwargs or {}))


def test_modes_and_transforms(both):
    q, kv, idx, scales = _prefill(2, 64, 256, 2048, "bf16", "fp8")
    call = lambda q=q: api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales)      # noqa: E731
    plain = call()

    def counted():
        with _Count() as mode:
            r = call()
        assert mode.n == 3                                                            # out, lse, workspace
        return r
    short, general, took = both(counted)
    assert took == [False]
    _same(short, plain)
    _same(general, plain)
    ones = torch.ones(3, device=DEV)
    short, general, took = both(lambda: torch.func.vmap(lambda x: (call(), x)[0], out_dims=(None, None))(ones))
    _same(short, plain)
    _same(general, plain)
    for f in (lambda: torch.func.vmap(lambda x: call(x))(torch.stack([q, q])), lambda: torch.func.grad(lambda x: call(x)[0].float().sum())(q),
              lambda: torch.func.jvp(call, (q,), (q,)), lambda: torch.func.grad(lambda x: call()[0].float().sum() + x.sum())(ones)):
        for way in (_lib.host(), None):
            with pytest.MonkeyPatch.context() as m:
                m.setattr(_lib, "_host", way)
                with pytest.raises(RuntimeError, match="data pointer"):
                    f()


def test_capture(both):
    q, kv, idx, scales = _prefill(2, 64, 1024, 4096, "bf16", "fp8")
    q2 = _prefill(2, 64, 1024, 4096, "e4m3", "fp8")[0].float().to(torch.bfloat16).mul_(2.0 ** -6)

    def captured():
        x = q.clone()
        api.sparse_prefill(x, kv, idx, synth.SM_SCALE, **scales)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out, lse = api.sparse_prefill(x, kv, idx, synth.SM_SCALE, **scales)
        x.copy_(q2)
        g.replay()
        torch.cuda.synchronize()
        return out.clone(), lse.clone()
    short, general, took = both(captured)
    assert took == [True, True]
    _same(short, general)
    _same(short, api.sparse_prefill(q2, kv, idx, synth.SM_SCALE, **scales))


def test_threads_on_streams_of_their_own():
    q, kv, idx, scales = _prefill(8, 64, 1024, 4096, "bf16", "fp8")
    xi = [x.to(DEV) for x in synth.make_indexer_operands(8, 3000, 32, seed=8)]
    r = torch.randn((24, 16, 576), device=DEV).to(torch.bfloat16)
    kr = torch.randn((20000, 576), device=DEV).to(torch.bfloat16)

    def all_three():
        return (*api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales), api.lite_topk(*xi, 64, 2992).sort(dim=1).values,
                *api.dsv4_c128a_bf16(r, kr[:156], kr, 19976, synth.SM_SCALE))
    want, got = all_three(), [None] * 4
    torch.cuda.synchronize()

    def work(i):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            results = [all_three() for _ in range(50)]
        stream.synchronize()
        got[i] = results
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    for results in got:
        for x in results:
            _same(x, want)


def test_other_threads_run_during_calls():
    q, kv, idx, scales = _prefill(2, 64, 256, 2048, "bf16", "fp8")
    keep, n, done = [], [0], threading.Event()

    def count():
        while not done.is_set():
            n[0] += 1
            time.sleep(0)
    interval, thread = sys.getswitchinterval(), threading.Thread(target=count)
    api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales)
    try:
        sys.setswitchinterval(1000.0)      # nobody has to hand over: the calls do so of their own accord
        thread.start()
        before = n[0]
        for _ in range(200):
            keep.append(api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales))
        assert n[0] > before
    finally:
        done.set()
        sys.setswitchinterval(interval)
        thread.join()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="two GPUs")
def test_another_current_device(both):
    q, kv, idx, scales = _prefill(2, 64, 256, 2048, "bf16", "fp8")
    with torch.cuda.device(1):
        short, general, took = both(lambda: api.sparse_prefill(q, kv, idx, synth.SM_SCALE, **scales))
    assert took == [False]
    _same(short, general)
