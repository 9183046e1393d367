"""A bounded device-side wait that runs out, on one GPU and without any fault: a sharded engine (rank 0 of 2) is given
a loopback exchange in which the other rank's share never arrives.  Every exchange wait then reaches its (shortened)
bound, the kernels carry on, the step finishes, and the host reads PI_ERR_TIMEOUT from the status word.  After the shares
are filled in from the host the same engine runs clean steps again: the context was never lost."""
import numpy as np
import pytest

from powerinfer_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_exchange_wait_runs_out_and_the_engine_stays_usable():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200 import engine
    from powerinfer_b200._lib import lib
    spec = synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=synth.Q4_0, n_layer=2, d=512, n_ff=2048, n_head=4, n_head_kv=2, rank=64,
                           firing=0.15, seed=41)
    eng = engine.DecodeEngine(spec, synth.build_model(spec), max_batch=1, n_ranks=2, rank=0)
    eng.setup_exchange_loopback()
    eng.set_wait_cycles(2_000_000)                 # about a millisecond per wait instead of a second
    for step in range(3):                          # plain launch, graph capture, graph replay
        eng.decode([7], [step])
        rc = lib.pi_engine_status(eng.handle, eng.st)
        assert rc == 5, (step, rc, lib.pi_last_error())        # PI_ERR_TIMEOUT
        assert b"exchange" in lib.pi_last_error()
    assert lib.pi_engine_status(eng.handle, eng.st) == 0       # reported once, then cleared
    eng.fill_peer_shares()
    logits, amax = eng.decode([7], [3])
    eng.status()                                               # clean
    assert np.isfinite(logits).all() and int(amax[0]) == int(logits[0].argmax())
    eng.close()


def _sharded(max_batch, wtype=synth.Q4_0):
    from powerinfer_b200 import engine
    spec = synth.ModelSpec(arch=synth.ARCH_LLAMA, wtype=wtype, n_layer=2, d=512, n_ff=2048, n_head=4, n_head_kv=2, rank=64, firing=0.15, seed=41)
    eng = engine.DecodeEngine(spec, synth.build_model(spec), max_batch=max_batch, n_ranks=2, rank=0)
    eng.setup_exchange_loopback()
    return eng


def _status_word(eng):
    """The engine's status word as a view of its workspace: the one word that pi_engine_status clears after a wait ran out."""
    from powerinfer_b200._lib import lib
    eng.set_wait_cycles(1_000_000)
    eng.decode([7], [0])
    off = (-eng.ws.data_ptr()) % 256
    words = eng.ws[off:off + (eng.ws.numel() - off) // 4 * 4].view(torch.int32)
    before = words.clone()
    assert lib.pi_engine_status(eng.handle, eng.st) == 5
    at = (before != words).nonzero()
    assert at.numel() == 1 and before[at].item() == 1
    return words[at.item():at.item() + 1]


@pytest.mark.parametrize("wtype", [synth.F16, synth.Q4_0])
def test_a_late_rank_runs_out_only_the_exchange_wait_of_a_batch(wtype):
    """The dense products of a batch are resident while the exchange before them still polls.  Their own bounded waits start when it is
    over, however long it took."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200._lib import lib
    eng = _sharded(3, wtype)
    word = _status_word(eng)
    eng.set_wait_cycles(300_000_000)               # about 0.15 s per exchange
    for step in range(3):                          # plain launch, graph capture, graph replay
        eng.decode([7, 8, 9], [step] * 3)
        assert word.item() == 1
        assert lib.pi_engine_status(eng.handle, eng.st) == 5 and b"exchange" in lib.pi_last_error()
    eng.close()


@pytest.mark.parametrize("bit", [2, 4, 8, 16])
def test_every_status_bit_is_reported(bit):
    """Each kind of kernel sets a bit of its own when a wait runs out; the host puts it there in a kernel's place."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from powerinfer_b200._lib import lib
    eng = _sharded(1)
    word = _status_word(eng)
    word.fill_(bit)
    torch.cuda.synchronize()
    assert lib.pi_engine_status(eng.handle, eng.st) == 5 and b"status %d" % bit in lib.pi_last_error()
    assert (b"one-launch step" in lib.pi_last_error()) == (bit == 8) and (b"weight-streaming" in lib.pi_last_error()) == (bit != 8)
    assert word.item() == 0 and lib.pi_engine_status(eng.handle, eng.st) == 0
    eng.close()
