"""The one-launch decode step (csrc/pi_step.cu) over the forms it takes.  Against the launch sequence it replaces: graphs, weight types, head
sizes, ragged sizes, rows in pieces, contexts beyond one pass of the attention, nearly all and few neurons active.  Against the CPU checker:
pieces of unequal length, exactly no and exactly every neuron active, more rows than one pass of the axpy, of the mask scan or of a phase's
sums takes.  (What its ring plan does at all other sizes is walked on the CPU: test_step_plan_cpu.py.)

Two correct implementations differ in the order of their sums, which flips roundings of activations between the nodes (FP16, or the int8 of
Q8_0): the bounds are those of perf/cases.py for whole steps, relative in the 2-norm: 3e-3 (FP16 weights), 3e-2 (Q4_0).  The predictors lie
far from the threshold against the launch sequence, so both choose the same neurons; the CPU checker is given the engine's choice."""
import ctypes
import os
import subprocess
import threading

import numpy as np
import pytest

from powerinfer_b200 import synth

pytestmark = pytest.mark.gpu


def _case(arch, wtype, n_layer, d, n_ff, n_head, n_head_kv, rank, n_vocab, n_ctx, firing, pos, batch=1):
    return dict(kind="decode", arch=arch, wtype=wtype, n_layer=n_layer, d=d, n_ff=n_ff, n_head=n_head, n_head_kv=n_head_kv, rank=rank, n_vocab=n_vocab,
                n_ctx=n_ctx, firing=firing, batch=batch, pos=pos)


CASES = {
    # d just above the narrowest model, a rank of one unit, a vocabulary that divides nothing, the first position
    "llama_q4_narrow": _case("llama", "q4_0", 3, 768, 2016, 6, 6, 8, 509, 96, 0.2, 0),
    "llama_f16_gqa_64": _case("llama", "f16", 2, 1024, 1312, 16, 1, 1368, 1001, 160, 0.3, 158),
    "llama_f16_pieces": _case("llama", "f16", 2, 5120, 3456, 40, 8, 488, 777, 128, 0.1, 77),
    "llama_q4_pieces": _case("llama", "q4_0", 1, 12544, 1600, 98, 7, 256, 515, 64, 0.2, 63),
    "llama_f16_wide": _case("llama", "f16", 1, 9216, 1376, 72, 8, 520, 300, 64, 0.2, 20),
    # rows just above a ring slot's usual size: whole, and in two pieces that fill the slot
    "llama_f16_whole_rows": _case("llama", "f16", 1, 4352, 1376, 34, 2, 96, 300, 64, 0.2, 20),
    "falcon_f16_two_pieces": _case("falcon", "f16", 1, 8448, 1376, 66, 22, 96, 300, 64, 0.2, 20),
    "llama_q4_whole_rows": _case("llama", "q4_0", 1, 13312, 1376, 104, 8, 96, 300, 64, 0.2, 20),
    "falcon_q4": _case("falcon", "q4_0", 2, 1280, 3904, 20, 5, 552, 600, 200, 0.15, 130),
    "falcon_f16": _case("falcon", "f16", 3, 2048, 4096, 32, 2, 144, 901, 96, 0.1, 50),
    "opt_f16": _case("opt", "f16", 2, 1536, 4032, 12, 12, 200, 1003, 128, 0.1, 90),
    "bamboo_q4": _case("bamboo", "q4_0", 2, 2560, 7776, 20, 20, 208, 1500, 96, 0.2, 33),
    "bamboo_f16": _case("bamboo", "f16", 2, 1024, 2080, 8, 4, 808, 640, 96, 0.2, 95),
    "long_context": _case("llama", "q4_0", 2, 1024, 2048, 8, 2, 64, 512, 3584, 0.2, 3583),
    "all_active": _case("llama", "q4_0", 2, 1024, 8192, 8, 2, 64, 512, 64, 0.9999, 5),
    "few_active": _case("llama", "f16", 2, 1024, 4096, 8, 2, 64, 512, 64, 1e-5, 5),
    "row_of_a_batch_engine": _case("llama", "f16", 2, 1024, 2048, 8, 2, 64, 512, 64, 0.2, 9, batch=3),
}


def _engine(case, one, seed=5):
    cases = pytest.importorskip("perf.cases")
    old = os.environ.get("PI_STEP")
    os.environ["PI_STEP"] = "1" if one else "0"
    try:
        return cases._prepare_engine(case, seed)["eng"]
    finally:
        if old is None:
            del os.environ["PI_STEP"]
        else:
            os.environ["PI_STEP"] = old


def _steps(eng, case, n=3):
    out = []
    for i in range(n):
        pos = max(0, min(case["pos"] - (n - 1) + i, case["n_ctx"] - 1))
        logits, ids = eng.decode([(7 + 31 * i) % case["n_vocab"]], [pos])
        out.append(np.array(logits[0]))
        assert int(ids[0]) == int(np.argmax(out[-1]))
    eng.status()
    return np.stack(out)


def _close(got, want, wtype):
    rel = np.linalg.norm(got.astype(np.float64) - want) / np.linalg.norm(want.astype(np.float64))
    assert np.isfinite(got).all() and rel <= (3e-2 if wtype == "q4_0" else 3e-3), rel


@pytest.mark.parametrize("name", list(CASES))
def test_step_matches_the_launch_sequence(name):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    case = CASES[name]
    ref = _engine(case, False)
    want = _steps(ref, case)
    assert ref.launches() > 1
    keys, values, total = ref.k_cache.float().cpu().numpy(), ref.v_cache.float().cpu().numpy(), ref.active_total()
    ref.close()
    eng = _engine(case, True)
    got = _steps(eng, case)
    assert eng.launches() == 1
    _close(got, want, case["wtype"])
    _close(eng.k_cache.float().cpu().numpy(), keys, case["wtype"])
    _close(eng.v_cache.float().cpu().numpy(), values, case["wtype"])
    assert eng.active_total() == total
    # the same bits again, fed from the device as well as from the host, and with the predictor's logits kept
    eng.enable_trace()
    again = _steps(eng, case)
    assert np.array_equal(again[-1], got[-1])
    assert (eng.predictor_trace(1)[:, 0] != 0).any()
    pos = max(0, min(case["pos"], case["n_ctx"] - 1))
    eng.set_inputs_device([(7 + 31 * 2) % case["n_vocab"]], [pos])
    eng.step_device(1)
    torch.cuda.synchronize()
    assert np.array_equal(eng.device_view("logits", 1)[0].cpu().numpy(), got[-1])
    eng.status()
    eng.close()


# rows whose pieces have unequal lengths, and predictors of such ranks
UNEVEN = {
    "f16_d_8320": dict(wtype=synth.F16, d=8320, n_ff=1088, n_head=65, n_head_kv=5, rank=72),
    "f16_d_8512": dict(wtype=synth.F16, d=8512, n_ff=1056, n_head=133, n_head_kv=7, rank=64),
    "f16_rank_4104": dict(wtype=synth.F16, d=1024, n_ff=2080, n_head=8, n_head_kv=2, rank=4104),
    "q4_rank_1552": dict(wtype=synth.Q4_0, d=5120, n_ff=1184, n_head=40, n_head_kv=8, rank=1552),
    "q4_rank_3080": dict(wtype=synth.Q4_0, d=4096, n_ff=1376, n_head=32, n_head_kv=4, rank=3080),
}


def _against_checker(spec, steps=2, launches=None):
    """Steps of an engine and of the CPU checker under the engine's own active sets: predictor logits and logits.  Active neurons of each step."""
    from oracle import pio
    from powerinfer_b200 import engine
    tensors = synth.build_model(spec)
    eng = engine.DecodeEngine(spec, tensors, max_batch=1)
    eng.enable_trace()
    om = pio.OracleModel(spec, tensors)
    wtype = "q4_0" if spec.wtype == synth.Q4_0 else "f16"
    active = []
    for pos in range(steps):
        tok = (7 + 31 * pos) % spec.n_vocab
        logits, ids = eng.decode([tok], [pos])
        got = eng.predictor_trace(1)[:, 0]
        want, pred = om.decode_imposed(tok, pos, got)
        _close(got, pred, wtype)
        _close(logits[0], want, wtype)
        assert int(ids[0]) == int(np.argmax(logits[0]))
        active.append(int((got >= spec.threshold).sum()))
    if launches is not None:
        assert eng.launches() == launches
    eng.status()
    eng.close()
    om.close()
    return active


@pytest.mark.parametrize("name", list(UNEVEN))
def test_rows_cut_into_unequal_pieces(name):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    _against_checker(synth.ModelSpec(arch=synth.ARCH_LLAMA, n_layer=1, n_vocab=320, n_ctx=64, firing=0.2, seed=3, **UNEVEN[name]))


# the threshold below or above every logit.  every_*: more than 512 rows in a group of the axpy, 2 and 4 mask words a thread (more than 16384,
# 32768 neurons), more rows of the gather, of fc2 and of the lm head in a CTA than have room for their sums at once
EXTREMES = {
    "none_llama_q4": (0, dict(arch=synth.ARCH_LLAMA, wtype=synth.Q4_0, d=1024, n_ff=2048, n_head=8, n_head_kv=2, rank=64, n_vocab=320)),
    "none_llama_f16": (0, dict(arch=synth.ARCH_LLAMA, wtype=synth.F16, d=1024, n_ff=2048, n_head=8, n_head_kv=2, rank=64, n_vocab=320)),
    "none_falcon_q4": (0, dict(arch=synth.ARCH_FALCON, wtype=synth.Q4_0, d=1024, n_ff=2048, n_head=16, n_head_kv=2, rank=64, n_vocab=320)),
    "none_opt_f16": (0, dict(arch=synth.ARCH_OPT, wtype=synth.F16, d=1024, n_ff=2048, n_head=8, n_head_kv=8, rank=64, n_vocab=320)),
    "every_q4_20480": (20480, dict(arch=synth.ARCH_LLAMA, wtype=synth.Q4_0, d=1024, n_ff=20480, n_head=8, n_head_kv=2, rank=64, n_vocab=320)),
    "every_q4_40960": (40960, dict(arch=synth.ARCH_FALCON, wtype=synth.Q4_0, d=1024, n_ff=40960, n_head=8, n_head_kv=2, rank=64, n_vocab=320)),
    "every_q4_wide": (4096, dict(arch=synth.ARCH_LLAMA, wtype=synth.Q4_0, d=8192, n_ff=4096, n_head=64, n_head_kv=8, rank=64, n_vocab=320)),
    "every_f16_65536": (65536, dict(arch=synth.ARCH_LLAMA, wtype=synth.F16, d=768, n_ff=65536, n_head=6, n_head_kv=2, rank=4096, n_vocab=100000)),
}


@pytest.mark.parametrize("name", list(EXTREMES))
def test_no_neuron_and_every_neuron_active(name):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    active, spec = EXTREMES[name]
    assert _against_checker(synth.ModelSpec(n_layer=1, n_ctx=64, seed=9, threshold=-1e30 if active else 1e30, **spec), launches=1) == [active, active]


@pytest.mark.parametrize("name", ["llama_q4_narrow", "llama_f16_gqa_64", "llama_f16_pieces", "falcon_q4", "opt_f16", "bamboo_q4", "all_active"])
def test_waits_that_run_out_are_reported_and_the_next_step_is_right(name):
    """A bound of one cycle: the first copying warp that has to wait gives up and ends the others' waits.  With larger bounds it is one that
    waits longer, in the middle of the step (for a slot, for the rows of the gather), or none.  The step comes to its end, the host reads the
    status, and the next step with the usual bound gives the bits of a run without any of this."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200._lib import lib
    case = CASES[name]
    eng = _engine(case, True)
    want = _steps(eng, case)
    pos = max(0, min(case["pos"], case["n_ctx"] - 1))
    for cycles in (1, 2000, 4000, 7000, 10000, 15000, 20000, 30000, 45000, 70000, 100000):
        for _ in range(5):
            eng.set_wait_cycles(cycles)
            eng.set_inputs_device([(7 + 31 * 2) % case["n_vocab"]], [pos])
            eng.step_device(1)
            rc = lib.pi_engine_status(eng.handle, eng.st)
            assert rc == 5 or (rc == 0 and cycles > 1), cycles                                              # PI_ERR_TIMEOUT
            assert (int(eng.device_view("argmax", 1)[0]) == -1) == (rc == 5)
            assert rc == 0 or b"status 8" in lib.pi_last_error()
            assert lib.pi_engine_status(eng.handle, eng.st) == 0                                            # reported once
        eng.set_wait_cycles(0)
        assert np.array_equal(_steps(eng, case), want)
    assert eng.launches() == 1
    eng.close()


def test_a_step_that_gives_up_is_an_error_of_the_call():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200._lib import lib
    case = CASES["llama_f16_gqa_64"]
    eng = _engine(case, True)
    want = _steps(eng, case)
    for want_logits in (True, False):
        eng.set_wait_cycles(1)
        with pytest.raises(RuntimeError, match="ran out"):
            eng.decode([3], [case["pos"]], want_logits=want_logits)      # (what it leaves in the cache is overwritten below)
        assert int(eng.h_argmax[0]) == -1
        assert lib.pi_engine_decode_host(eng.handle, eng.h_tokens.data_ptr(), eng.h_pos.data_ptr(), 1, None, None, eng.st) == 5
        eng.set_wait_cycles(0)
        eng.status()                                              # the call has reported it
        assert np.array_equal(_steps(eng, case), want)
    eng.close()


HOLD = r"""
#include <cuda_runtime.h>
__global__ void hold(unsigned long long ns) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
    for (int i = 0; i < 10000000; i++) {
        __nanosleep(1000);
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
        if (t1 - t0 >= ns) break;
    }
}
extern "C" int hold_sm(unsigned long long ns, void * stream) {
    if (cudaFuncSetAttribute(hold, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) return 1;
    hold<<<1, 32, 200 * 1024, (cudaStream_t)stream>>>(ns);
    return (int)cudaGetLastError();
}
"""


def test_a_kernel_of_another_stream_may_hold_an_sm(tmp_path):
    """An SM is taken for 0.4 s, far longer than a wait's bound of about 20 ms: the step waits for it and is right."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import build
    src, so = tmp_path / "hold.cu", tmp_path / "libhold.so"
    src.write_text(HOLD)
    subprocess.run([build.NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC", "-o", str(so), str(src)], check=True)
    hold = ctypes.CDLL(str(so)).hold_sm
    hold.argtypes = [ctypes.c_ulonglong, ctypes.c_void_p]
    case = CASES["llama_f16_gqa_64"]
    eng = _engine(case, True)
    want = _steps(eng, case)
    eng.set_wait_cycles(40_000_000)
    other = torch.cuda.Stream()
    for _ in range(2):
        assert hold(400_000_000, other.cuda_stream) == 0
        got = _steps(eng, case)                                   # (asserts a clean status)
        other.synchronize()
        assert np.array_equal(got, want)
    eng.close()


def test_a_stream_with_a_part_of_the_device_runs_the_launch_sequence():
    """All CTAs of the step run at once; where a stream has too few SMs for them (a green context), the launch sequence takes the step."""
    torch = pytest.importorskip("torch")
    driver = pytest.importorskip("cuda.bindings.driver")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200._lib import check, lib
    case = CASES["llama_f16_gqa_64"]
    eng = _engine(case, False)
    want = _steps(eng, case)
    eng.close()
    eng = _engine(case, True)
    one = _steps(eng, case)
    assert eng.launches() == 1

    def ok(r):
        if r[0] != driver.CUresult.CUDA_SUCCESS:
            pytest.skip(f"no green context here: {r[0]}")
        return r[1:] if len(r) > 2 else (r[1] if len(r) == 2 else None)

    dev = ok(driver.cuDeviceGet(0))
    sms = ok(driver.cuDeviceGetDevResource(dev, driver.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups, _, _ = ok(driver.cuDevSmResourceSplitByCount(1, sms, 0, 32))
    green = ok(driver.cuGreenCtxCreate(ok(driver.cuDevResourceGenerateDesc([groups[0]], 1)), dev, driver.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(driver.cuGreenCtxStreamCreate(green, driver.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    for i in range(3):                                            # plain launch, graph capture, graph replay
        eng.h_tokens[0], eng.h_pos[0] = (7 + 31 * 2) % case["n_vocab"], case["pos"]
        check(lib.pi_engine_decode_host(eng.handle, eng.h_tokens.data_ptr(), eng.h_pos.data_ptr(), 1, eng.h_logits.data_ptr(), eng.h_argmax.data_ptr(), int(stream)))
        assert eng.launches() > 1
        _close(eng.h_logits[0].numpy(), want[-1], case["wtype"])
    assert np.array_equal(_steps(eng, case)[-1], one[-1]) and eng.launches() == 1
    eng.close()
    ok(driver.cuStreamDestroy(stream))
    ok(driver.cuGreenCtxDestroy(green))


def test_a_profiled_step_is_held_until_its_launches_are_queued():
    """The stream is held while the host queues the launch sequence: 12 us a launch, 12 ms where none was counted yet, whatever a step
    launches by itself."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import time
    eng = _engine(_case("llama", "f16", 24, 768, 2048, 6, 6, 64, 512, 64, 0.2, 3), True)
    eng.decode([5], [3])
    assert eng.launches() == 1
    for least in (lambda n: 1000, lambda n: n):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        ms, n = eng.profile_step(1)
        assert time.perf_counter() - t0 >= least(n) * 12e-6
        assert n > 8 * 24 and ms["qkv"] > 0 and eng.launches() == 1
    eng.status()
    eng.close()


def test_a_step_inside_a_captured_graph():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    case = CASES["llama_f16_gqa_64"]
    eng = _engine(case, True)
    want = _steps(eng, case)
    graph = torch.cuda.CUDAGraph()
    pos = max(0, min(case["pos"], case["n_ctx"] - 1))
    eng.set_inputs_device([(7 + 31 * 2) % case["n_vocab"]], [pos])
    with torch.cuda.graph(graph, stream=eng.stream, capture_error_mode="thread_local"):
        eng.step_device(1)
    for _ in range(3):
        eng.device_view("logits", 1).zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(eng.device_view("logits", 1)[0].cpu().numpy(), want[-1])
    eng.status()
    del graph
    eng.close()


def test_steps_of_two_engines_in_two_threads():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    cs = [CASES["llama_f16_gqa_64"], CASES["falcon_q4"]]
    engs = [_engine(c, True) for c in cs]
    want = [_steps(e, c) for e, c in zip(engs, cs)]
    bad = []

    def work(e, c, w):
        try:
            for _ in range(30):
                if not np.array_equal(_steps(e, c), w):
                    bad.append("other bits")
        except Exception as ex:
            bad.append(repr(ex))

    ts = [threading.Thread(target=work, args=a) for a in zip(engs, cs, want)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad, bad[:3]
    [e.close() for e in engs]
