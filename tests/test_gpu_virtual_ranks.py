"""GPU, one device: the passes of several ranks through mok.functional, each rank driven by a host thread of this process
on buffers of its own, one at a time.  No kernel waits for another one: where ranks meet on the device in earnest (the
barrier kernel), the threads meet on the host instead.  Row movement, schedules and peer addresses are those of real ranks."""
import threading

import pytest
import torch

from oracle import mok_oracle as O
from tests.helpers import BF16_REL_L2, MXFP8_REL_L2, rel_l2
from tests.test_gpu_layer import GRAD_NAMES

pytestmark = pytest.mark.gpu

CFG = dict(T=512, H=256, I=256, E=8, W=2, K=2)
CAPACITY = 4096                     # skewed routing gives one of the ranks 2560 rows, the other 256


def run_ranks(monkeypatch, dev, ranks, *, macrobatch, minibatch, mxfp8):
    """Forward + backward of every rank: per rank a dict of output, gradients and schedule; and the profile slots used."""
    import mok
    F, L = mok.functional, mok._lib
    W, (T, H), K = len(ranks), ranks[0].x.shape, ranks[0].topk_experts.shape[1]
    El = ranks[0].w_routed_gate.shape[0]
    cfg = F.MoKConfig(minibatch_size=minibatch, macrobatch_size=macrobatch, schedule_capacity_multiplier=2.0,
                      all_gather_top_experts_chunk_bytes=16)
    shapes = dict(x_buffer=((T, H), torch.bfloat16), combine_buffer=((T * K, H), torch.bfloat16),
                  d_y_buffer=((T, H), torch.bfloat16), d_x_routed_buffer=((T * K, H), torch.bfloat16),
                  router_weight_buffer=((T, K), torch.float32), d_router_weight_buffer=((T, K), torch.float32),
                  all_gather_top_experts_buffer=((W, T, K), torch.int32), barrier_buffer=((1,), torch.int32))
    buffers = [{n: torch.zeros(s, dtype=dt, device=dev) for n, (s, dt) in shapes.items()} for _ in range(W)]
    ptrs = {n: [b[n].data_ptr() for b in buffers] for n in shapes}
    with_ptrs = set(shapes) - {"all_gather_top_experts_buffer"}
    workspaces = []
    for r, b in enumerate(buffers):
        L.register_all_gather_peers(b["all_gather_top_experts_buffer"].data_ptr(), ptrs["all_gather_top_experts_buffer"])
        workspaces.append(F.MoKWorkspace(
            group_name="virtual", ep_rank=r, ep_size=W, device=dev, num_local_tokens=T, hidden_size=H, topk=K,
            schedule_capacity=CAPACITY, all_gather_top_experts_buffer_multicast_ptr=0, barrier_buffer_multicast_ptr=0,
            barrier_target=torch.zeros(1, dtype=torch.int32, device=dev), **b,
            **{n + "_handle": None for n in shapes}, **{n + "_ptrs": ptrs[n] for n in with_ptrs}))
    meet, turn = threading.Barrier(W, timeout=60), threading.Lock()

    def barrier(_ws):
        torch.cuda.synchronize(dev)
        turn.release()
        try:
            meet.wait()
        finally:
            turn.acquire()
    monkeypatch.setattr(F, "_barrier", barrier)
    results, errors = [None] * W, []

    def rank_main(r):
        turn.acquire()
        try:
            torch.cuda.set_device(dev)
            me, ws = ranks[r], workspaces[r]
            d = lambda t: t.to(dev)  # noqa: E731
            x, rw = d(me.x), d(me.router_weights)
            w = [d(t) for t in (me.w_shared_gate, me.w_shared_up, me.w_shared_down, me.w_routed_gate, me.w_routed_up,
                                me.w_routed_down)]
            fw = bw = w
            if mxfp8:
                qg, qu, qd = (mok.ops.mxfp8_quantize(t, True, True) for t in w[3:])
                fw = w[:3] + [(qg[0], qg[1]), (qu[0], qu[1]), (qd[0], qd[1])]
                bw = w[:3] + [tuple(qg), tuple(qu), (qd[2], qd[3])]
            sched = F.build_schedule(ws, cfg, d(me.topk_experts), num_local_experts=El)
            out, ctx = F.forward(cfg, ws, sched, x, rw, *fw)
            barrier(ws)
            grads = F.backward(cfg, ws, sched, ctx, d(me.d_output), x, rw, *bw)
            torch.cuda.synchronize(dev)
            results[r] = dict(zip(GRAD_NAMES, grads), output=out, schedule=sched)
        except BaseException as e:  # noqa: BLE001  (reported by the main thread; the others leave the barrier at once)
            errors.append(e)
            meet.abort()
        finally:
            turn.release()

    L.check(L.mok_profile_enable(1), "profile")
    L.profile_collect()
    try:
        threads = [threading.Thread(target=rank_main, args=(r,)) for r in range(W)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize(dev)
        slots = L.profile_collect()
    finally:
        L.mok_profile_enable(0)
        for b in buffers:
            L.unregister_all_gather_peers(b["all_gather_top_experts_buffer"].data_ptr())
    if errors:
        raise next((e for e in errors if not isinstance(e, threading.BrokenBarrierError)), errors[0])
    assert mok.last_status(dev)[0] == 0, mok.last_status(dev)
    return results, slots


@pytest.mark.parametrize("mxfp8", [False, True])
@pytest.mark.parametrize("zipf", [None, 1.2])
def test_two_ranks_whole_windows_and_chunks(cuda_device, monkeypatch, mxfp8, zipf):
    """Windows below two minibatches are moved in one piece, larger ones in chunks beside the GEMMs: both give the oracle's
    results, the same bytes, and the launches of several ranks (no stage shared by the two kinds of expert)."""
    ranks = [O.make_rank_inputs(r, seed=61, zipf_s=zipf, **CFG) for r in range(2)]
    ref = O.layer_forward_backward(ranks, device_rounding=True, mxfp8=mxfp8, capacity=CAPACITY)
    tol = MXFP8_REL_L2 if mxfp8 else BF16_REL_L2
    got = {}
    for macro, mini in ((4096, 4096), (4096, 256), (1024, 1024), (1024, 256)):
        got[macro, mini], slots = run_ranks(monkeypatch, cuda_device, ranks, macrobatch=macro, minibatch=mini, mxfp8=mxfp8)
        assert not any("joint" in name for name in slots), slots
        for r, res in enumerate(got[macro, mini]):
            for name in ("peer_rank", "peer_token_idx", "num_tokens", "tokens_per_expert"):
                assert (ref[r][name] == getattr(res["schedule"], name).cpu().numpy()).all(), (macro, mini, r, name)
            for name in ("output",) + GRAD_NAMES:
                assert rel_l2(ref[r][name].float(), res[name].float()) < tol, (macro, mini, r, name)
    for macro, mini in ((4096, 256), (1024, 256)):
        for whole, cut in zip(got[macro, macro], got[macro, mini]):
            for name in ("output",) + GRAD_NAMES:
                assert torch.equal(whole[name], cut[name]), (macro, name)
