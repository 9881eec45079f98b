"""The native front of the entry points (csrc/fast_path.cpp) takes the ordinary call of every mode and
gives what the wrapper's own way gives; whatever is not ordinary it leaves to the wrapper, unlaunched."""

import ctypes
import subprocess
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

MODES = ("w8a8-mxfp8", "w4a4-mxfp4", "w4a4-nvfp4")


@pytest.fixture(scope="module")
def hq():
    import halops_b200

    return halops_b200


@pytest.fixture(scope="module")
def native(hq):
    from halops_b200 import _native

    _native.load_fast_path()
    return _native


class Sub(torch.Tensor):
    pass


def _bytes(*tensors):
    return [t.view(torch.uint8) for t in tensors]


@pytest.mark.parametrize("mode", MODES)
@pytest.mark.parametrize("m,n,k", [(1, 128, 256), (130, 256, 512), (256, 384, 1024)], ids=lambda v: str(v))
def test_same_results_both_ways(hq, native, monkeypatch, mode, m, n, k):
    g = torch.Generator().manual_seed(m + n)
    a = torch.randn([m, k], generator=g).to(torch.bfloat16).cuda()
    b = torch.randn([n, k], generator=g).to(torch.float16).cuda()
    alpha = torch.full([1], 0.5, device="cuda") if mode == "w4a4-nvfp4" else None
    results = []
    for front in (native.fast_path, native._NoFastPath):
        monkeypatch.setattr(native, "fast_path", front)
        aq, sfa = hq.group_wise_quant(a, mode)
        bq, sfb = hq.group_wise_quant(b, mode)
        out = torch.empty([m, n], dtype=torch.bfloat16, device="cuda")
        hq.dense_gemm(aq, bq, sfa, sfb, out, alpha=alpha, mode=mode)
        rows = _bytes(*hq.rms_norm_quant(a, a[0].contiguous(), 1e-5, False))
        results.append(_bytes(aq, sfa, bq, sfb) + [out] + rows)
    for x, y in zip(*results):
        assert x.shape == y.shape and torch.equal(x, y)


def test_what_it_takes_and_what_it_leaves(hq, native):
    f = native.fast_path
    x = torch.randn([64, 256], device="cuda").to(torch.bfloat16)
    q, sf = f.group_wise_quant(x, "w8a8-mxfp8", True, True, None, None)
    assert f.group_wise_quant(x, "w8a8-mxfp8", True, True, q, sf)[0] is q
    w, sfw = hq.group_wise_quant(torch.randn([128, 256], device="cuda").to(torch.bfloat16))
    out = torch.full([64, 128], 7.0, dtype=torch.bfloat16, device="cuda")

    def dense(x=q, w=w, sf=sf, sfw=sfw, out=out, bias=None, alpha=None, mode="w8a8-mxfp8", pdl=True, epilogue=0):
        return f.dense_gemm(x, w, sf, sfw, out, bias, alpha, -1, mode, pdl, epilogue, None, 4.0, 25.0)

    untouched = out.clone()
    left = [dense(x=q.cpu()), dense(x=q.as_subclass(Sub)), dense(sf=sf.flatten()[:-1]), dense(w=w[:, :128]), dense(pdl=None),
            dense(mode="w4a4-nvfp4"), dense(mode="bf16"), dense(epilogue=1), dense(out=out.float()), dense(alpha=sf),
            dense(bias=torch.zeros([128], dtype=torch.bfloat16, device="cuda")), dense(out=out.t()),
            f.group_wise_quant(x, "w8a8-mxfp8", 1, True, None, None), f.group_wise_quant(x.t(), "w8a8-mxfp8", True, True, None, None),
            f.group_wise_quant(x.float(), "w8a8-mxfp8", True, True, None, None),
            f.group_wise_quant(x, "w8a8-mxfp8", True, True, sf, None), f.rms_norm_quant(x, x[0, :128], 1e-6, True, True)]
    assert left == [None] * len(left)
    with torch.overrides.TorchFunctionMode():
        assert dense() is None
    torch.cuda.synchronize()
    assert torch.equal(out, untouched)
    assert dense() is True and not torch.equal(out, untouched)


def test_grouped(hq, native, monkeypatch):
    e, rows, n, k = 3, 64, 128, 256
    x, sfa = hq.group_wise_quant(torch.randn([e * rows, k], device="cuda").to(torch.bfloat16))
    w, sfb = (torch.stack(t) for t in zip(*(hq.group_wise_quant(torch.randn([n, k], device="cuda").to(torch.bfloat16))
                                            for _ in range(e))))
    counts = torch.tensor([5, 0, 64], dtype=torch.int32, device="cuda")
    ids = torch.arange(e, dtype=torch.int32, device="cuda").repeat_interleave(rows)
    results = []
    for front in (native.fast_path, native._NoFastPath):
        monkeypatch.setattr(native, "fast_path", front)
        out = torch.zeros([2, e * rows, n], dtype=torch.bfloat16, device="cuda")
        hq.group_masked_gemm(x, w, sfa, sfb, counts, out[0], max_m_per_expert=rows)
        hq.group_contiguous_gemm(x, w, sfa, sfb, ids, out[1])
        results.append(out)
        with pytest.raises(RuntimeError, match="input M must equal num_experts"):
            hq.group_masked_gemm(x, w, sfa, sfb, counts, out[0], max_m_per_expert=2 * rows)
    assert torch.equal(*results)


ALLOCATOR = """
#include <cuda_runtime.h>
#include <sys/types.h>
extern "C" int PyGILState_Check(void);
static int calls, locked;
extern "C" void* count_alloc(ssize_t size, int, cudaStream_t) {
    ++calls;
    locked += PyGILState_Check();
    void* p = nullptr;
    return cudaMalloc(&p, size) == cudaSuccess ? p : nullptr;
}
extern "C" void count_free(void* p, ssize_t, int, cudaStream_t) { cudaFree(p); }
extern "C" int count_calls(void) { return calls; }
extern "C" int count_locked(void) { return locked; }
"""


@pytest.mark.parametrize("entry", ["group_wise_quant", "rms_norm_quant"])
def test_outputs_are_allocated_without_the_interpreter_lock(hq, native, tmp_path, entry):
    """An allocation may wait for the device (a full card, a stream that a host function in Python holds up):
    other Python threads must be able to run meanwhile."""
    from halops_b200 import build

    source, lib = tmp_path / "alloc.cpp", tmp_path / "alloc.so"
    source.write_text(ALLOCATOR)
    cuda = build.cuda_root()
    subprocess.run(["g++", "-shared", "-fPIC", "-o", lib, source, f"-I{cuda}/include", f"-L{cuda}/lib64", "-lcudart"], check=True)
    x = torch.randn([64, 256], device="cuda").to(torch.bfloat16)
    weight = x[0].contiguous()
    pool = torch.cuda.MemPool(torch.cuda.memory.CUDAPluggableAllocator(str(lib), "count_alloc", "count_free").allocator())
    counts = ctypes.CDLL(str(lib))
    with torch.cuda.use_mem_pool(pool):
        if entry == "group_wise_quant":
            outputs = native.fast_path.group_wise_quant(x, "w8a8-mxfp8", True, True, None, None)
        else:
            outputs = native.fast_path.rms_norm_quant(x, weight, 1e-6, True, True)
    assert outputs is not None
    torch.cuda.synchronize()
    assert counts.count_calls() > 0 and counts.count_locked() == 0
    del outputs


def test_two_threads(hq, native):
    """Each thread on a stream of its own, with its own inputs, outputs and weights: what one thread alone gets."""
    g = torch.Generator().manual_seed(4)
    sizes = [(8, 1024, 512), (200, 256, 384)]
    jobs = []
    for m, n, k in sizes:
        x = torch.randn([m, k], generator=g).to(torch.bfloat16).cuda()
        w, sfw = hq.group_wise_quant(torch.randn([n, k], generator=g).to(torch.bfloat16).cuda())
        jobs.append((x, w, sfw, n))

    def chain(job):
        x, w, sfw, n = job
        outs = []
        for _ in range(50):
            q, sf = hq.group_wise_quant(x)
            out = torch.empty([x.size(0), n], dtype=torch.bfloat16, device="cuda")
            hq.dense_gemm(q, w, sf, sfw, out)
            outs.append(out)
        return outs

    expected = [chain(job)[0] for job in jobs]
    torch.cuda.synchronize()
    results = [None] * len(jobs)

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            results[i] = chain(jobs[i])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert hq.device_status() == 0
    for want, outs in zip(expected, results):
        assert outs is not None and all(torch.equal(want, out) for out in outs)


class Recorder:
    """The native front, noting whether it took each call."""

    def __init__(self, front):
        self.front, self.took = front, []

    def __getattr__(self, name):
        def call(*args):
            result = getattr(self.front, name)(*args)
            self.took.append(result is not None)
            return result
        return call


def _both_ways(native, monkeypatch, calls):
    """The results of ``calls`` through the native front, which must take every call, and through the wrappers."""
    recorder = Recorder(native.load_fast_path())
    results = []
    for front in (recorder, native._NoFastPath):
        monkeypatch.setattr(native, "fast_path", front)
        results.append([t.view(torch.uint8) for call in calls for t in call()])
        torch.cuda.synchronize()
    assert recorder.took and all(recorder.took), recorder.took
    for x, y in zip(*results):
        assert x.shape == y.shape and torch.equal(x, y)


def test_dense_options_both_ways(hq, native, monkeypatch):
    m, n, k = 256, 512, 384
    g = torch.Generator().manual_seed(21)
    wide = torch.randn([m, k + 128], generator=g).to(torch.bfloat16).cuda()
    a, sfa = hq.group_wise_quant(wide[:, :k].contiguous())
    b, sfb = hq.group_wise_quant((torch.randn([n, k], generator=g) * 0.1).to(torch.bfloat16).cuda())
    bias = torch.randn([n], generator=g).to(torch.bfloat16).cuda()

    def dense(**kw):
        out = torch.zeros([m, n + 64], dtype=torch.bfloat16, device="cuda")
        hq.dense_gemm(a, b, sfa, sfb, out[:, :n], **kw)  # (rows of the output are strided)
        return [out]

    def situ(**kw):
        out = torch.zeros([m, n // 2], dtype=torch.float8_e4m3fn, device="cuda")
        sf = torch.zeros([m, n // 64], dtype=torch.uint8, device="cuda")
        hq.dense_gemm(a, b, sfa, sfb, out, epilogue=hq.EpilogueOp.SituQuant, output_sf=sf, **kw)
        return [out, sf]

    _both_ways(native, monkeypatch, [
        lambda: hq.group_wise_quant(wide[:, :k]), lambda: hq.group_wise_quant(wide[:, :k], use_swizzle=False, use_pdl=False),
        lambda: hq.rms_norm_quant(wide[:, :k], bias[:k]),
        lambda: dense(), lambda: dense(bias=bias), lambda: dense(epilogue=hq.EpilogueOp.Sigmoid, sm_count=64), lambda: dense(use_pdl=2),
        lambda: situ(), lambda: situ(bias=bias, situ_linear_beta=None), lambda: situ(situ_beta=2, use_pdl=False)])


@pytest.mark.parametrize("mode", MODES + ("w4a8-mxfp4",))
def test_grouped_options_both_ways(hq, native, monkeypatch, mode):
    e, rows, n, k = 3, 128, 256, 512
    g = torch.Generator().manual_seed(22)
    act, wgt = ("w8a8-mxfp8", "w4a4-mxfp4") if mode == "w4a8-mxfp4" else (mode, mode)
    x, sfa = hq.group_wise_quant(torch.randn([e * rows, k], generator=g).to(torch.bfloat16).cuda(), act)
    w, sfb = hq.group_wise_quant((torch.randn([e * n, k], generator=g) * 0.1).to(torch.bfloat16).cuda(), wgt)
    w, sfb = w.view(e, n, -1), sfb.view(e, n, -1)
    alpha = torch.tensor([0.5, 1.0, 2.0], device="cuda") if mode == "w4a4-nvfp4" else None
    biases = [None] + ([torch.randn([e, n], generator=g).to(torch.bfloat16).cuda()] if mode == "w8a8-mxfp8" else [])
    counts = torch.tensor([5, 0, 128], dtype=torch.int32, device="cuda")
    ids = torch.tensor([0] * 64 + [1] * 192 + [2] * 128, dtype=torch.int32, device="cuda")

    def masked(bias):
        out = torch.zeros([e * rows, n + 8], dtype=torch.bfloat16, device="cuda")
        hq.group_masked_gemm(x, w, sfa, sfb, counts, out[:, :n], bias, alpha, rows, mode=mode)
        return [out]

    def contiguous(bias):
        out = torch.zeros([e * rows, n], dtype=torch.bfloat16, device="cuda")
        hq.group_contiguous_gemm(x, w, sfa, sfb, ids, out, bias, alpha, mode=mode)
        return [out]

    _both_ways(native, monkeypatch, [lambda f=f, b=b: f(b) for f in (masked, contiguous) for b in biases])
