"""Submissions go to the senders from the caller's thread where their targets are known, through the manager's thread where not."""
import random
import threading

import pytest
import torch

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer, ReqMeta

L, T, TOK, NB = 2, 16, 64, 128


@pytest.mark.parametrize("seed, cap", [(1, 0), (2, 1), (3, 2)])
def test_threads_submit_while_targets_come_and_go(ops, seed, cap):
    """Three threads send frozen requests to three workers while a fourth evicts targets down to `cap`: every request arrives once."""
    src = [torch.randint(0, 256, (NB * T * TOK,), dtype=torch.uint8) for _ in range(L)]
    dst = [[torch.zeros_like(t) for t in src] for _ in range(3)]
    kw = dict(num_kv_heads=1, cache_shape=2)
    srvs = [KVTransferServer("D%d|0|1" % i, 1, 0, 0, T * TOK, TOK, "fake://", dst[i], [PT.TCP], **kw) for i in range(3)]
    cli = KVTransferClient("P|0|1", 1, 0, 0, T * TOK, TOK, "fake://", src, [PT.TCP], **kw)
    per_thread, stop, sent, errors = 20, threading.Event(), [], []

    def send(k):
        rng = random.Random(seed * 10 + k)
        try:
            for i in range(per_thread):
                d, b = rng.randrange(3), 1 + k * per_thread + i
                m = ReqMeta()
                m.dst_inst, m.dst_worker, m.reqid = "D%d|0|1" % d, 0, "r%d.%d" % (k, i)
                m.seen_tokens, m.new_tokens = 0, T
                m.src_block_ids, m.dst_block_ids, m.dst_worker_info = [[b]], [[b]], srvs[d].worker_info()
                cli.start_req_send([m], 1000 * k + i)
                sent.append((d, b))
        except Exception as ex:  # noqa: BLE001
            errors.append(ex)

    def evict():
        while not stop.is_set():
            cli._c.target_try_shrink(cap)

    try:
        threads = [threading.Thread(target=send, args=(k,)) for k in range(3)]
        evictor = threading.Thread(target=evict)
        for t in threads + [evictor]:
            t.start()
        for t in threads:
            t.join()
        stop.set()
        evictor.join()
        assert not errors
        cli.drain()
        assert cli.inflight() == 0 and cli.failed_batches() == 0 and len(sent) == 3 * per_thread
        half = T * TOK // 2           # K and V of a block lie in the two halves of the cache
        for d in range(3):
            got = {b for w, b in sent if w == d}
            for layer in range(L):
                a, z = src[layer].view(2, NB, half), dst[d][layer].view(2, NB, half)
                for b in range(NB):
                    assert torch.equal(z[:, b], a[:, b]) if b in got else not bool(z[:, b].any())
        cli._c.target_try_shrink(0)
        assert cli._c.target_size() == 0
    finally:
        cli.drain()
        del cli
        for s in srvs:
            s.stop()
