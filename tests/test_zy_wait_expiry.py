"""The failure path of the device-side waits, exercised without hanging or faulting anything: one CTA of a row-slab launch
is told (by a host option) to keep its z values to itself, so every consumer's bounded poll runs out of its (shortened)
budget, records its code in the scratch's status words and leaves through the common exit. The call returns, the status
says which wait gave up, reset() re-arms the scratch and the next call is bit-identical to a clean one.
Counterpart in the reference: the bounded polls that record a code in Diag[4095] (csrc/biloco_gemm.cu:1149-1151, 1288).
Collected late on purpose: it leaves the library's process-wide options at their defaults, but a failure here should not
hide the results of the other tests."""
import time

import numpy as np
import pytest
import torch

from oracle import biloco_oracle as orc
from tests.gpu_util import dev_problem

pytestmark = pytest.mark.gpu

ST_Z = 105          # status code of the z poll (csrc/fused_cfg.cuh)


@pytest.mark.parametrize("M", [1, 4])        # (the four-row kernel has a z poll of its own: two vectors per round trip)
def test_z_poll_runs_out_and_scratch_recovers(M):
    from biloco_b200 import _lib, kernel
    lib = _lib.load()
    K, N, R = 1024, 1024, 512              # (every CTA owns at least three ranks)
    assert 7 in kernel.supported_modes(M, N, K, R)
    p = orc.random_problem(M, K, N, R, scales="random", seed=11)
    t = dev_problem(p)
    g = kernel.BiLoCoGemm(t["W"], t["W_sf"], t["alpha"], t["V_packed"], t["U_packed"], t["S"], M=M, mode=7)

    def run():
        y = g(t["A_pad"], t["A_sf"], t["X"]).view(-1, N)[:M].clone()
        torch.cuda.synchronize()
        return y

    clean = run()
    assert g.status()[0] == 0
    try:
        lib.biloco_b200_set_option(_lib.OPT_WAIT_BUDGET_US, 2000)
        lib.biloco_b200_set_option(_lib.OPT_SKIP_PUBLISH, 0)          # CTA 0 computes its z slice and does not publish it
        t0 = time.perf_counter()
        run()
        dt = time.perf_counter() - t0
    finally:
        lib.biloco_b200_set_option(_lib.OPT_SKIP_PUBLISH, -1)
        lib.biloco_b200_set_option(_lib.OPT_WAIT_BUDGET_US, 0)         # back to the default budget
    st = g.status()
    assert st[0] == ST_Z, f"expected the z poll's code in the status word, got {st[:4]}"
    assert 0 <= st[1] < 148 * 2 and st[2] == g.epoch                   # the block that gave up first, the call's epoch
    assert dt < 1.0, f"the call took {dt:.3f} s: a wait did not honour its budget"
    # the status word is sticky until the scratch's head is cleared
    g.reset()
    assert g.status()[0] == 0
    again = run()
    assert g.status()[0] == 0
    assert torch.equal(again.view(torch.int16), clean.view(torch.int16)), "the call after reset() differs from a clean one"
    again = run()
    assert torch.equal(again.view(torch.int16), clean.view(torch.int16))


@pytest.mark.parametrize("M", [8, 16, 32])
def test_batch_z_poll_runs_out_and_later_launches_are_right(M):
    """The same for five to 32 rows: one CTA keeps its partial sums of z to itself, the CTAs that add them up give up within the
    budget. The launches that follow on the SAME scratch, without reset(), are right: no value of the failed launch or of the
    one before it passes for a later one's."""
    from biloco_b200 import _lib, kernel
    lib = _lib.load()
    K, N, R = 1024, 1024, 512
    ps = [orc.random_problem(M, K, N, R, scales="random", seed=11 + i) for i in range(2)]
    ts = [dev_problem(p) for p in ps]
    t = ts[0]
    g = kernel.BiLoCoGemm(t["W"], t["W_sf"], t["alpha"], t["V_packed"], t["U_packed"], t["S"], M=M, mode=2)

    def run(i=0):                            # (the second activation goes with the first problem's weights)
        y = g(ts[i]["A_pad"], ts[i]["A_sf"], ts[i]["X"]).view(-1, N)[:M].clone()
        torch.cuda.synchronize()
        return y

    clean = [run(0), run(1)]
    assert g.status()[0] == 0
    for before in range(2):                  # (either parity of the launch count)
        run(1)
        try:
            lib.biloco_b200_set_option(_lib.OPT_WAIT_BUDGET_US, 2000)
            lib.biloco_b200_set_option(_lib.OPT_SKIP_PUBLISH, 0)
            t0 = time.perf_counter()
            run(0)
            dt = time.perf_counter() - t0
        finally:
            lib.biloco_b200_set_option(_lib.OPT_SKIP_PUBLISH, -1)
            lib.biloco_b200_set_option(_lib.OPT_WAIT_BUDGET_US, 0)
        st = g.status()
        assert st[0] == ST_Z and st[2] > 0 and dt < 1.0, (st[:4], dt)
        for i in (0, 1, 0):
            assert torch.equal(run(i).view(torch.int16), clean[i].view(torch.int16)), (before, i)
        if before == 0:
            run(1)
    g.reset()
    assert g.status()[0] == 0
    assert torch.equal(run(0).view(torch.int16), clean[0].view(torch.int16)) and g.status()[0] == 0


@pytest.mark.parametrize("R", [0, 96])
def test_prompt_wait_runs_out_and_the_layer_says_so(R):
    """More than 32 rows: one CTA of the z launch and of the GEMM does not fetch its operands, its waits run out of the budget. The layer's
    own status words say so until they are cleared, another layer's do not; the calls after it are right."""
    import ctypes
    from biloco_b200 import _lib
    from biloco_b200.layer import BiLoCoLinear
    lib = _lib.load()
    K, N, rows = 1024, 264, 140
    ops = BiLoCoLinear.synthetic(K, N, max(R, 1), "cuda", seed=4).export_operands()
    if R == 0:
        ops["V_packed"], ops["U_packed"], ops["S"] = ops["V_packed"][:0], ops["U_packed"][:0], ops["S"][:0]
    layer, other = BiLoCoLinear.from_operands(ops), BiLoCoLinear.from_operands(ops)
    x = torch.randn(rows, K, device="cuda").to(torch.bfloat16)
    clean = layer(x)
    assert torch.equal(other(x), clean) and layer.status() == [0] * 16
    try:
        lib.biloco_b200_set_option(_lib.OPT_WAIT_BUDGET_US, 2000)
        lib.biloco_b200_set_option(_lib.OPT_SKIP_PUBLISH, 0)
        t0 = time.perf_counter()
        layer(x)
        torch.cuda.synchronize()
        dt = time.perf_counter() - t0
    finally:
        lib.biloco_b200_set_option(_lib.OPT_SKIP_PUBLISH, -1)
        lib.biloco_b200_set_option(_lib.OPT_WAIT_BUDGET_US, 0)
    st = layer.status()
    assert st[0] in (121, 122) and st[1] == 0 and dt < 1.0, (st[:4], dt)
    assert torch.equal(other(x), clean) and other.status() == [0] * 16
    assert torch.equal(layer(x), clean) and layer.status()[0] == st[0]
    layer.reset_status()
    assert layer.status() == [0] * 16
    words = (ctypes.c_int32 * 16)()
    for want in (st[0], 0):                  # (the device-wide words: read and cleared)
        assert lib.biloco_b200_prompt_status(words, torch.cuda.current_stream().cuda_stream) == 0 and words[0] == want


def test_peer_allreduce_wait_runs_out_and_reports(lib):
    """The peer all-reduce polls its own receive buffer for the peers' words with a time budget. Here a 'group' of two
    with nobody behind rank 1 (its buffer is a second local allocation that nothing reads or writes back): the poll runs
    out, the kernel records it and returns, the context stays usable, and a later launch on the same GPU is unaffected."""
    import ctypes
    world, slot = 2, 1024
    nbytes = lib.biloco_b200_peer_buffer_bytes(world, slot)
    bufs = []
    for _ in range(2):
        p, h = ctypes.c_void_p(), (ctypes.c_ubyte * 64)()
        assert lib.biloco_b200_peer_buffer_create(nbytes, ctypes.byref(p), h) == 0
        bufs.append(p.value)
    table = torch.tensor(bufs, dtype=torch.int64, device="cuda")
    status = torch.zeros(16, dtype=torch.int32, device="cuda")
    part = torch.ones(512, device="cuda")
    out = torch.zeros(512, device="cuda", dtype=torch.bfloat16)
    assert lib.biloco_b200_set_option(5, 2000) == 0              # BILOCO_OPT_WAIT_BUDGET_US
    try:
        rc = lib.biloco_b200_peer_allreduce(part.data_ptr(), None, out.data_ptr(), table.data_ptr(), status.data_ptr(), world, 0, 512, slot, 0,
                                            torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
    finally:
        lib.biloco_b200_set_option(5, 0)
    st = status.cpu().tolist()
    assert st[0] == 1 and st[2] == 1 and st[3] == 0, st            # gave up, in call 1, on rank 0
    assert (st[8] >> 20) == 1                                       # the call counter advanced all the same
    assert float((torch.ones(8, device="cuda") * 2).sum()) == 16.0   # the context still works
    for b in bufs:
        assert lib.biloco_b200_peer_buffer_destroy(b) == 0
