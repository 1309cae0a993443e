"""Several layers of a step in one launch: whatever the launches hold, every layer's bytes are those that the forward stream wrote
before it recorded the layer's event, and nothing outside the request's slots is written."""
import os
import subprocess
import sys
import time

import pytest
import torch

os.environ.setdefault("BLLM_KVTRANS_QUIET_ENV", "1")

from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer, ReqMeta
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


BLOCK = 64


class _Cache:
    """One rank's cache of a shape: its tensors, the sizes that the engine is told, and a request's bytes of a layer."""

    def __init__(self, shape, layers, blocks):
        self.mla = shape == CacheShape.DPSK_V32_SPARSE_MLA
        self.lay = AttnLayout(CacheShape.FLASH, blocks, BLOCK, 8, 128, 2)
        self.toks = [132, 656] if self.mla else [self.lay.token_bytes]
        self.layers = [[torch.zeros(blocks * BLOCK * t, dtype=torch.uint8, device=DEV) for t in self.toks] for _ in range(layers)]
        one = (lambda x: x) if self.mla else (lambda x: x[0])
        self.args = one([BLOCK * t for t in self.toks]), one(self.toks), "fake://", [one(t) for t in self.layers], [PT.NVLINK]
        self.kw = dict(num_kv_heads=1 if self.mla else 8, cache_shape=int(shape))

    def rows(self, layer, first, n):
        """Every token slot of blocks [first, first + n), one row each and tensor."""
        if not self.mla:
            v = self.lay.view(self.layers[layer][0], torch.int16)[first:first + n]     # [block, kv, slot, head, dim]
            return [v.movedim(1, 2).reshape(n * BLOCK, -1).view(torch.uint8)]
        return [t.view(-1, BLOCK * k)[first:first + n].reshape(n * BLOCK, k) for t, k in zip(self.layers[layer], self.toks)]


@pytest.mark.parametrize("host_gap_s", [0.0, 0.002])
@pytest.mark.parametrize("shape", [CacheShape.FLASH, CacheShape.DPSK_V32_SPARSE_MLA])
@pytest.mark.parametrize("layers, tokens", [(1, 16), (2, 1), (13, 75), (13, 3001), (33, 700)])
def test_every_layer_carries_what_was_recorded(layers, tokens, shape, host_gap_s):
    """75 tokens: 4 MiB hold every layer.  3001: half of the rest per launch.  host_gap_s: a forward thread slower than the
    sender, so that it waits for layers; without it the layers are all recorded long before the GPU has produced them."""
    n = -(-tokens // BLOCK)
    src, dst = _Cache(shape, layers, 2 * n + 2), _Cache(shape, layers, 2 * n + 2)
    srv = KVTransferServer("D|0|1", 1, 0, 0, *dst.args, **dst.kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, *src.args, **src.kw)
    try:
        fwd = torch.cuda.Stream()
        big = torch.empty(1 << 26, dtype=torch.uint8, device=DEV)
        for step in (1, 2, 3):
            sb, db = list(range(1, n + 1)), list(range(n + 1, 2 * n + 1))
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, tokens, True, sb, db, srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            with torch.cuda.stream(fwd):
                for layer in range(layers):
                    big.fill_(layer)                     # the layer is produced "late"
                    for t in src.layers[layer]:
                        t.fill_((7 * layer + 31 * step) % 251 + 1)
                    cli.record_event(layer, fwd)
                    time.sleep(host_gap_s)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                v = (7 * layer + 31 * step) % 251 + 1
                for got in dst.rows(layer, n + 1, n):
                    assert int(got[:tokens].min()) == int(got[:tokens].max()) == v
                    assert dst.mla or not bool(got[tokens:].any())
                for untouched in dst.rows(layer, 0, n + 1):
                    assert not bool(untouched.any())
    finally:
        cli.drain()
        del cli
        srv.stop()


def test_layers_recorded_on_the_current_stream_whichever_it_is():
    """record_event() without a stream takes the current one, also when that changes from step to step."""
    layers, n = 6, 5
    src, dst = _Cache(CacheShape.FLASH, layers, 2 * n + 2), _Cache(CacheShape.FLASH, layers, 2 * n + 2)
    srv = KVTransferServer("D|0|1", 1, 0, 0, *dst.args, **dst.kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, *src.args, **src.kw)
    try:
        streams = [torch.cuda.Stream(), torch.cuda.default_stream(), torch.cuda.Stream()]
        big = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
        for step in range(1, 7):
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, n * BLOCK, True, list(range(n)), list(range(n + 1, 2 * n + 1)),
                                 srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            with torch.cuda.stream(streams[step % 3]):
                for layer in range(layers):
                    big.fill_(layer)
                    src.layers[layer][0].fill_(10 * step + layer)
                    cli.record_event(layer)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                got = dst.rows(layer, n + 1, n)[0]
                assert int(got.min()) == int(got.max()) == 10 * step + layer
    finally:
        cli.drain()
        del cli
        srv.stop()


@pytest.mark.parametrize("layers, tokens", [(6, 100), (9, 3001)])
def test_layers_recorded_on_several_streams_of_one_step(layers, tokens):
    """Even layers are produced late on one stream, odd ones at once on another: the event of the last layer of a launch says
    nothing about the others."""
    n = -(-tokens // BLOCK)
    src, dst = _Cache(CacheShape.FLASH, layers, 2 * n + 2), _Cache(CacheShape.FLASH, layers, 2 * n + 2)
    srv = KVTransferServer("D|0|1", 1, 0, 0, *dst.args, **dst.kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, *src.args, **src.kw)
    try:
        slow, fast = torch.cuda.Stream(), torch.cuda.Stream()
        big = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
        for step in (1, 2, 3):
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, tokens, True, list(range(n)), list(range(n + 1, 2 * n + 1)),
                                 srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                with torch.cuda.stream(fast if layer % 2 else slow):
                    if layer % 2 == 0:
                        for _ in range(4):
                            big.fill_(layer)
                    src.layers[layer][0].fill_(40 * step + layer)
                    cli.record_event(layer)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                got = dst.rows(layer, n + 1, n)[0][:tokens]
                assert int(got.min()) == int(got.max()) == 40 * step + layer
    finally:
        cli.drain()
        del cli
        srv.stop()


@pytest.mark.parametrize("proto", [PT.NVLINK, PT.SHM])
@pytest.mark.parametrize("shape", [CacheShape.FLASH, CacheShape.DPSK_V32_SPARSE_MLA])
@pytest.mark.parametrize("recorded", [1, 5])
def test_a_step_flushed_before_its_last_layers_still_waits_for_those_recorded(recorded, shape, proto):
    """The layers behind the last one recorded keep the events (and the bytes) of the step before: those events are long
    complete and say nothing about the layers that this step recorded."""
    layers, n = 9, 3
    src, dst = _Cache(shape, layers, 2 * n + 2), _Cache(shape, layers, 2 * n + 2)
    args = lambda c: c.args[:4] + ([proto],)  # noqa: E731
    srv = KVTransferServer("D|0|1", 1, 0, 0, *args(dst), **dst.kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, *args(src), **src.kw)
    try:
        fwd = torch.cuda.Stream()
        big = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
        value = [0] * layers
        for step, upto in ((1, layers), (2, recorded), (3, recorded), (4, layers), (5, recorded)):
            cli.submit_req_send2("D|0|1", 0, "r%d" % step, 0, n * BLOCK, True, list(range(n)), list(range(n + 1, 2 * n + 1)),
                                 srv.worker_info(), stepid=step)
            cli.start_send_step(step, 1)
            with torch.cuda.stream(fwd):
                for layer in range(upto):
                    for _ in range(4):
                        big.fill_(layer)
                    value[layer] = 20 * step + layer
                    for t in src.layers[layer]:
                        t.fill_(value[layer])
                    cli.record_event(layer)
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                for got in dst.rows(layer, n + 1, n):
                    assert int(got.min()) == int(got.max()) == value[layer], (step, layer)
    finally:
        cli.drain()
        del cli
        srv.stop()


@pytest.mark.parametrize("shape", [CacheShape.FLASH, CacheShape.DPSK_V32_SPARSE_MLA])
@pytest.mark.parametrize("layers, blocks", [(9, 30), (34, 70)])
def test_a_frozen_send_waits_for_the_layers_of_the_step_before_it(layers, blocks, shape):
    """The step that produced the data used two streams, or recorded some of the layers only.  (34, 70) is 595 MiB of
    the attention cache and goes out in several launches, the others in one."""
    src, dst = _Cache(shape, layers, blocks + 1), _Cache(shape, layers, blocks + 1)
    srv = KVTransferServer("D|0|1", 1, 0, 0, *dst.args, **dst.kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, *src.args, **src.kw)
    try:
        slow, fast = torch.cuda.Stream(), torch.cuda.Stream()
        big = torch.empty(1 << 28, dtype=torch.uint8, device=DEV)
        value = [0] * layers
        # (streams of even and odd layers, layers recorded)
        for step, (even, upto) in enumerate([(slow, layers), (fast, layers), (slow, layers), (fast, layers - 2), (slow, layers)], 1):
            cli.start_send_step(step, 1)
            for layer in range(upto):
                with torch.cuda.stream(fast if layer % 2 else even):
                    if layer % 2 == 0:
                        for _ in range(4):
                            big.fill_(layer)
                    value[layer] = 40 * step + layer
                    for t in src.layers[layer]:
                        t.fill_(value[layer])
                    cli.record_event(layer)
            cli.flush_send_step()
            m = ReqMeta()
            m.dst_inst, m.dst_worker, m.reqid, m.dst_worker_info = "D|0|1", 0, "m%d" % step, srv.worker_info()
            m.seen_tokens, m.new_tokens = 0, blocks * BLOCK
            m.src_block_ids, m.dst_block_ids = [list(range(blocks))], [list(range(1, blocks + 1))]
            cli.start_req_send([m], step)
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                for got in dst.rows(layer, 1, blocks):
                    assert int(got.min()) == int(got.max()) == value[layer], (step, layer)
    finally:
        cli.drain()
        del cli
        srv.stop()


@pytest.mark.parametrize("walk", [1, 0])
def test_walk_and_descriptor_launches_of_layers_recorded_on_several_streams(walk):
    """The two ways of moving a cache of several tensors a layer; the switch between them is read once in a process."""
    script = """
import torch
import test_step_launches_gpu as t
t.several_streams(t.CacheShape.DPSK_V32_SPARSE_MLA, 9, 3001)
print("ok")
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, BLLM_KVTRANS_NVLINK_WALK=str(walk), PYTHONPATH=os.pathsep.join([root, os.path.join(root, "tests")]))
    r = subprocess.run([sys.executable, "-c", script], env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("ok\n"), r.stderr[-3000:]


def several_streams(shape, layers, tokens):
    """Even layers late on one stream, odd ones at once on another.  The request joins the step when all of them have been
    recorded, so that every launch takes as many as it can."""
    n = -(-tokens // BLOCK)
    src, dst = _Cache(shape, layers, n + 1), _Cache(shape, layers, n + 1)
    srv = KVTransferServer("D|0|1", 1, 0, 0, *dst.args, **dst.kw)
    cli = KVTransferClient("P|0|1", 1, 0, 0, *src.args, **src.kw)
    try:
        slow, fast = torch.cuda.Stream(), torch.cuda.Stream()
        big = torch.empty(1 << 30, dtype=torch.uint8, device=DEV)
        for step in (1, 2, 3):
            cli.start_send_step(step, 1)
            for layer in range(layers):
                with torch.cuda.stream(fast if layer % 2 else slow):
                    for _ in range(0 if layer % 2 else 6):
                        big.fill_(layer)
                    for t in src.layers[layer]:
                        t.fill_(40 * step + layer)
                    cli.record_event(layer)
            m = ReqMeta()
            m.dst_inst, m.dst_worker, m.reqid, m.dst_worker_info = "D|0|1", 0, "m%d" % step, srv.worker_info()
            m.seen_tokens, m.new_tokens = 0, tokens
            m.src_block_ids, m.dst_block_ids = [list(range(n))], [list(range(1, n + 1))]
            cli.start_send_substep(step, 1, [m])
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                for rows in dst.rows(layer, 1, n):
                    got = rows[:tokens]
                    assert int(got.min()) == int(got.max()) == 40 * step + layer, (step, layer)
    finally:
        cli.drain()
        del cli
        srv.stop()


@pytest.mark.parametrize("host_gap_s", [0.0, 0.001])
def test_one_step_towards_a_device_ordered_and_a_host_driven_destination(host_gap_s):
    """The host-driven one wants to follow the layers one by one; the other lets the thread that waits for them sleep."""
    layers, n = 12, 5
    src = _Cache(CacheShape.FLASH, layers, n + 1)
    dsts = [_Cache(CacheShape.FLASH, layers, n + 1) for _ in range(2)]
    protos = [PT.NVLINK, PT.SHM]
    srvs = [KVTransferServer("D%d|0|1" % i, 1, 0, 0, *(d.args[:4] + ([p],)), **d.kw) for i, (d, p) in enumerate(zip(dsts, protos))]
    cli = KVTransferClient("P|0|1", 1, 0, 0, *(src.args[:4] + (protos,)), **src.kw)
    try:
        fwd = torch.cuda.Stream()
        big = torch.empty(1 << 27, dtype=torch.uint8, device=DEV)

        def submit(i, step):
            cli.submit_req_send2("D%d|0|1" % i, 0, "r%d.%d" % (i, step), 0, n * BLOCK, True, list(range(n)), list(range(1, n + 1)),
                                 srvs[i].worker_info(), stepid=step)

        def meta(i, step):
            m = ReqMeta()
            m.dst_inst, m.dst_worker, m.reqid, m.dst_worker_info = "D%d|0|1" % i, 0, "s%d.%d" % (i, step), srvs[i].worker_info()
            m.seen_tokens, m.new_tokens, m.src_block_ids, m.dst_block_ids = 0, n * BLOCK, [list(range(n))], [list(range(1, n + 1))]
            return m

        for step in range(1, 9):
            late = step % 4                      # the host-driven destination: in the step from the start, or joins it later
            submit(0, step)
            if late == 0:
                submit(1, step)
            cli.start_send_step(step, 1)
            for layer in range(layers):
                with torch.cuda.stream(fwd):
                    big.fill_(layer)
                    src.layers[layer][0].fill_(16 * step + layer)
                    cli.record_event(layer)
                time.sleep(host_gap_s)
                if layer == (0, 0, layers // 2, layers - 1)[late] and late:
                    cli.start_send_substep(step, 1, [meta(1, step)])
            cli.flush_send_step()
            assert cli.wait_inflight(0, 30.0) and not cli.failed_batches()
            torch.cuda.synchronize()
            for layer in range(layers):
                for d in dsts:
                    got = d.rows(layer, 1, n)[0]
                    assert int(got.min()) == int(got.max()) == 16 * step + layer, (step, layer)
    finally:
        cli.drain()
        del cli
        for s in srvs:
            s.stop()
