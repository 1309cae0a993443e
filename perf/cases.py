"""The transfers this framework is used for, as timed cases.

Every case is one pass through a public entry point: an engine step of ``KVTransferClient`` towards a
``KVTransferServer`` (both caches on this GPU), a direct ``AttnTransfer``, or a save / load of the host-DRAM
``PinnedKVStore``.  Shapes are those of the model families in ``llumnix_kv_b200/models/kv_spec.py``.  A pass returns the
whole destination cache (as 64-bit words), so a missing or misplaced byte shows.
"""
from __future__ import annotations

import math
import os
import random
from typing import List

import torch

os.environ.setdefault("BLLM_KVTRANS_QUIET_ENV", "1")

from llumnix_kv_b200 import load_ops
from llumnix_kv_b200.kv_transfer_impl import KVTransferClient, KVTransferProtocolType as PT, KVTransferServer, ReqMeta
from llumnix_kv_b200.kvstore import PinnedKVStore
from llumnix_kv_b200.ops.layouts import AttnLayout, CacheShape
from llumnix_kv_b200.ops.p2d_attn import MODE_BF16_TO_MXFP8, MODE_COPY, MODE_MXFP8_TO_BF16, AttnTransfer, HeadMap, ReqChunk

DEV = "cuda:0"
BLOCK = 16            # tokens per block of the attention caches
DIM = 128
NHD, HND = int(CacheShape.FLASH), int(CacheShape.FLASHINFER)
MLA_TOKEN, MLA_BLOCK = (132, 656), 64     # indexer keys (128 e4m3 values and a scale), latent + rope
GDN_TOKEN, GDN_STATE = 2 * 2 * 256 * 2, 3 * 8192 * 2 + 16 * 128 * 128 * 4
GDN_BLOCK = ((GDN_STATE + GDN_TOKEN - 1) // GDN_TOKEN + 15) // 16 * 16     # tokens of a page that can hold that state


def listed() -> List[dict]:
    return [
        # a short chat turn leaves the prefill worker: latency of one engine step, hardly any bytes
        {"name": "turn", "kind": "push", "layers": 32, "tokens": 75, "reqs": 1, "seen": 0, "p_tp": 1, "d_tp": 1},
        # the headline: one 8192-token prompt of Llama-3-8B shape, FlashAttention NHD pages -> FlashInfer HND pages
        {"name": "prompt", "kind": "push", "layers": 32, "tokens": 8192, "reqs": 1, "seen": 0, "p_tp": 1, "d_tp": 1},
        # chunked prefill of several requests: chunks begin and end inside blocks, heads of a TP=2 prefill rank land in
        # the second half of a TP=1 decode worker's pages
        {"name": "chunks", "kind": "push", "layers": 32, "tokens": 3001, "reqs": 7, "seen": 37, "p_tp": 2, "d_tp": 1},
        # Llama-3-70B shape, a TP=4 prefill rank in bf16 -> its half of a TP=2 decode worker's block-scaled fp8 pages
        {"name": "quantise", "kind": "fp8", "layers": 80, "tokens": 6005, "reqs": 2, "seen": 0, "p_tp": 4, "d_tp": 2},
        # the other direction: block-scaled fp8 pages expanded into a bf16 cache
        {"name": "expand", "kind": "direct", "mode": MODE_MXFP8_TO_BF16, "src": HND, "dst": NHD, "layers": 32, "heads": 8,
         "tokens": 4003, "reqs": 3, "seen": 0},
        # one layer of a small batch by the kernel's own Python face: plan and launch
        {"name": "layer", "kind": "direct", "mode": MODE_COPY, "src": NHD, "dst": HND, "layers": 1, "heads": 8, "tokens": 333,
         "reqs": 4, "seen": 0},
        # a running request moves to another decode worker of the same layout
        {"name": "migrate", "kind": "migrate", "layers": 32, "tokens": 1111, "reqs": 1},
        # DeepSeek-V3.2 shape: 61 layers of two tensors, identical on both sides
        {"name": "mla", "kind": "mla", "layers": 61, "tokens": 20011, "reqs": 1},
        # Qwen3-Next shape: 12 physical tensors whose pages hold attention KV or the recurrent state of GDN layers
        {"name": "hybrid", "kind": "gdn", "layers": 12, "tokens": 30011, "reqs": 1},
        # prefix cache in host memory: blocks saved as they are, and loaded from block-scaled fp8 pages
        {"name": "save", "kind": "store", "load": False, "fp8": False, "layers": 32, "blocks": 24},
        {"name": "load_fp8", "kind": "store", "load": True, "fp8": True, "layers": 32, "blocks": 160},
        # two workers without peer access: gather, shared host memory, scatter
        {"name": "host_staged", "kind": "shm", "layers": 32, "tokens": 1024, "reqs": 1},
    ]


def _log(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["push", "push", "fp8", "direct", "direct", "migrate", "mla", "gdn", "store", "shm"])
    reqs = rng.randint(1, 8)
    if kind == "push":
        p_tp, d_tp = rng.choice([(1, 1), (2, 1), (1, 2), (4, 4), (8, 2)])
        return {"kind": kind, "layers": 32, "tokens": _log(rng, 16, 8192) + reqs, "reqs": reqs,
                "seen": rng.choice([0, 0, rng.randint(1, 500)]), "p_tp": p_tp, "d_tp": d_tp}
    if kind == "fp8":
        p_tp, d_tp = rng.choice([(4, 2), (4, 4), (8, 4), (2, 2)])
        return {"kind": kind, "layers": 80, "tokens": _log(rng, 64, 8192 if p_tp > 2 else 4096) + reqs, "reqs": reqs,
                "seen": rng.choice([0, 0, rng.randint(1, 500)]), "p_tp": p_tp, "d_tp": d_tp}
    if kind == "direct":
        mode = rng.choice([MODE_COPY, MODE_COPY, MODE_BF16_TO_MXFP8, MODE_MXFP8_TO_BF16])
        layers = rng.choice([1, 8, 32])
        src, dst = rng.choice([(NHD, HND), (HND, NHD), (NHD, NHD), (HND, HND), (int(CacheShape.RAGGED_FLASH), HND)])
        if mode == MODE_BF16_TO_MXFP8:
            dst = HND
        if mode == MODE_MXFP8_TO_BF16:
            src = HND
        return {"kind": kind, "mode": mode, "src": src, "dst": dst, "layers": layers, "heads": rng.choice([1, 2, 4, 8]),
                "tokens": _log(rng, 16, 8192) + reqs, "reqs": reqs, "seen": rng.choice([0, 0, rng.randint(1, 500)])}
    if kind == "migrate":
        return {"kind": kind, "layers": 32, "tokens": _log(rng, 1, 8192), "reqs": 1}
    if kind == "mla":
        return {"kind": kind, "layers": 61, "tokens": _log(rng, 64, 20000) + reqs, "reqs": reqs}
    if kind == "gdn":
        return {"kind": kind, "layers": 12, "tokens": _log(rng, 500, 30000) + reqs, "reqs": min(reqs, 4)}
    if kind == "store":
        return {"kind": kind, "load": rng.random() < 0.5, "fp8": rng.random() < 0.5, "layers": 32, "blocks": _log(rng, 2, 192)}
    return {"kind": kind, "layers": 32, "tokens": _log(rng, 32, 1500) + reqs, "reqs": reqs}


# ---- inputs ---------------------------------------------------------------------------------------------------
class _State:
    """What a worker keeps: caches, the open client and server, and the step's requests."""

    def __init__(self, case: dict, rng: random.Random, gen: torch.Generator):
        self.case, self.rng, self.gen = case, rng, gen
        self.cli = self.srv = self.store = self.xfer = None
        self.step_id = 100

    def __del__(self):
        if self.srv is not None:
            self.cli.drain()
            self.cli = None
            self.srv.stop()
        if self.store is not None:
            name = self.store_name
            self.store.close()
            load_ops().KvStore.unlink(name)


def _split(total: int, parts: int) -> List[int]:
    """`parts` positive prompt lengths of that sum, unequal as prompts are (the caches' sizes follow from them, so they depend
    on the case alone)."""
    rng, parts = random.Random(total * 31 + parts), min(parts, total)
    w = [rng.uniform(0.2, 1.0) for _ in range(parts)]
    lens = [max(1, int(total * x / sum(w))) for x in w]
    lens[0] += total - sum(lens)
    if lens[0] < 1:
        lens = [total // parts] * parts
        lens[0] += total - sum(lens)
    return lens


def _tables(s: _State, lens: List[int], block: int):
    """Block ids of every request on both sides, scattered over the pools as a running engine leaves them."""
    need = [-(-n // block) for n in lens]
    pool = sum(need) + sum(need) // 8 + 4
    a, b = s.rng.sample(range(1, pool), sum(need)), s.rng.sample(range(1, pool), sum(need))
    out, at = [], 0
    for n in need:
        out.append((a[at:at + n], b[at:at + n]))
        at += n
    return pool, out


def _normal_bf16(nbytes: int, gen: torch.Generator) -> torch.Tensor:
    return torch.empty(nbytes // 2, dtype=torch.bfloat16, device=DEV).normal_(generator=gen).view(torch.uint8)


def _bytes(nbytes: int, gen: torch.Generator) -> torch.Tensor:
    words = torch.empty(-(-nbytes // 8), dtype=torch.int64, device=DEV).random_(-2 ** 62, 2 ** 62, generator=gen)
    return words.view(torch.uint8)[:nbytes]


def _cut(flat: torch.Tensor, layers: int) -> List[torch.Tensor]:
    n = flat.numel() // layers
    return [flat[i * n:(i + 1) * n] for i in range(layers)]


def _engine(s: _State, src, dst, sizes, toks, src_shape, dst_shape, proto, p_tp=1, d_tp=1, p_rank=0, d_rank=0, dst_sizes=None,
            dst_toks=None, mx=False, **kw) -> None:
    inst = "D|0|%d" % d_tp
    s.dst_inst, s.d_rank = inst, d_rank
    s.srv = KVTransferServer(inst, d_tp, d_rank, d_rank, dst_sizes or sizes, dst_toks or toks, "fake://", dst, [proto],
                             cache_shape=dst_shape, mx_scaled=mx, **kw)
    s.winfo = s.srv.worker_info()
    s.cli = KVTransferClient("P|0|%d" % p_tp, p_tp, p_rank, p_rank, sizes, toks, "fake://", src, [proto], cache_shape=src_shape, **kw)


def _submit(s: _State) -> None:
    s.step_id += 1
    cli = s.cli
    for i, (sb, db, seen, new) in enumerate(s.reqs):
        cli.submit_req_send2(s.dst_inst, s.d_rank, "r%d.%d" % (s.step_id, i), seen, new, True, sb, db, s.winfo, stepid=s.step_id)
    cli.start_send_step(s.step_id, 1)
    for layer in range(s.case["layers"]):
        cli.record_event(layer)
    cli.flush_send_step()
    if not cli.wait_inflight(0, 30.0) or cli.failed_batches():
        raise RuntimeError("the transfer did not complete")


def _migrate(s: _State) -> None:
    s.step_id += 1
    metas = []
    for i, (sb, db, seen, new) in enumerate(s.reqs):
        m = ReqMeta()
        m.dst_inst, m.dst_worker, m.reqid = s.dst_inst, s.d_rank, "m%d.%d" % (s.step_id, i)
        m.seen_tokens, m.new_tokens = seen, new
        m.src_block_ids, m.dst_block_ids, m.dst_worker_info = [sb], [db], s.winfo
        metas.append(m)
    s.cli.start_req_send(metas, s.step_id)
    if not s.cli.wait_inflight(0, 30.0) or s.cli.failed_batches():
        raise RuntimeError("the transfer did not complete")


def _head_window(c: dict):
    """(heads of the prefill rank, of the decode rank, prefill rank, decode rank) of a pair of 8 KV heads."""
    p_heads, d_heads = 8 // c["p_tp"], 8 // c["d_tp"]
    if c["p_tp"] >= c["d_tp"]:
        p_rank = c["p_tp"] - 1
        return p_heads, d_heads, p_rank, p_rank * c["d_tp"] // c["p_tp"]
    return p_heads, d_heads, 0, c["d_tp"] // c["p_tp"] - 1


def prepare(case: dict, seed: int) -> _State:
    s = _State(case, random.Random(seed * 7919 + 1), torch.Generator(device=DEV).manual_seed(seed * 104729 + 5))
    kind, layers = case["kind"], case["layers"]
    if kind == "store":
        return _prepare_store(s)
    new = _split(case["tokens"], case["reqs"])
    seen = [case.get("seen", 0) * (1 + i) // 2 for i in range(len(new))]
    block = {"mla": MLA_BLOCK, "gdn": GDN_BLOCK}.get(kind, BLOCK)
    pool, tables = _tables(s, [a + b for a, b in zip(seen, new)], block)
    s.reqs = [(sb, db, a, b) for (sb, db), a, b in zip(tables, seen, new)]
    if kind in ("push", "fp8"):
        hp, hd, p_rank, d_rank = _head_window(case)
        src_l = AttnLayout(CacheShape.FLASH, pool, BLOCK, hp, DIM, 2)
        dst_l = AttnLayout(CacheShape.FLASHINFER, pool, BLOCK, hd, DIM, 1 if kind == "fp8" else 2, mx_scaled=kind == "fp8")
        s.src = _normal_bf16(layers * src_l.layer_bytes, s.gen)
        s.dst = torch.zeros(layers * dst_l.layer_bytes, dtype=torch.uint8, device=DEV)
        _engine(s, _cut(s.src, layers), _cut(s.dst, layers), src_l.block_bytes, src_l.token_bytes, NHD, HND, PT.NVLINK, case["p_tp"],
                case["d_tp"], p_rank, d_rank, dst_l.block_bytes, dst_l.token_bytes, kind == "fp8", num_kv_heads=8)
        s.go = _submit
    elif kind == "direct":
        mode, heads = case["mode"], case["heads"]
        lay = lambda shape, mx: AttnLayout(CacheShape(shape), pool, BLOCK, heads, DIM, 1 if mx else 2, mx_scaled=mx)  # noqa: E731
        src_l, dst_l = lay(case["src"], mode == MODE_MXFP8_TO_BF16), lay(case["dst"], mode == MODE_BF16_TO_MXFP8)
        if mode == MODE_MXFP8_TO_BF16:
            # e4m3 codes without NaN and exponents around one, as the quantiser writes them
            s.src = _bytes(layers * src_l.layer_bytes, s.gen)
            s.src &= 0xF7
            for flat in _cut(s.src, layers):
                sc = src_l.scale_view(flat)
                sc.copy_(torch.randint(115, 122, sc.shape, dtype=torch.uint8, device=DEV, generator=s.gen))
        else:
            s.src = _normal_bf16(layers * src_l.layer_bytes, s.gen)
        s.dst = torch.zeros(layers * dst_l.layer_bytes, dtype=torch.uint8, device=DEV)
        ptrs = lambda flat: [t.data_ptr() for t in _cut(flat, layers)]  # noqa: E731
        s.xfer = AttnTransfer(src_l, dst_l, ptrs(s.src), ptrs(s.dst), DEV, head_map=HeadMap(0, 0, heads), mode=mode)
        s.chunks = [ReqChunk(*r) for r in s.reqs]
        s.go = lambda st: st.xfer.launch(st.xfer.plan(st.chunks))
    elif kind in ("migrate", "shm"):
        shape = NHD if kind == "shm" else HND
        lay_ = AttnLayout(CacheShape(shape), pool, BLOCK, 8, DIM, 2)
        s.src = _normal_bf16(layers * lay_.layer_bytes, s.gen)
        s.dst = torch.zeros_like(s.src)
        _engine(s, _cut(s.src, layers), _cut(s.dst, layers), lay_.block_bytes, lay_.token_bytes, shape, shape,
                PT.SHM if kind == "shm" else PT.NVLINK, num_kv_heads=8)
        s.go = _migrate if kind == "migrate" else _submit
    else:
        # several tensors per layer, or pages of several kinds: one flat buffer per side, cut into the cache tensors
        if kind == "mla":
            toks, shape, kw = list(MLA_TOKEN), int(CacheShape.DPSK_V32_SPARSE_MLA), dict(num_kv_heads=1)
        else:
            toks, shape = [GDN_TOKEN], int(CacheShape.QWEN3_NEXT_FLASH)
            kw = dict(num_kv_heads=2, num_gdn_layers=3, conv_state_shape=[1, 3, 8192], ssm_state_shape=[1, 16, 128, 128],
                      gdn_conv_channel_dims=[2048, 2048, 4096], gdn_conv_elem_size=2, gdn_ssm_elem_size=4)
            # one page per GDN layer group and request holds its recurrent state, beside the attention pages
            extra = 3 * len(s.reqs)
            a, b = s.rng.sample(range(pool, pool + extra), extra), s.rng.sample(range(pool, pool + extra), extra)
            pool += extra
            s.reqs = [([[a[3 * i]], [a[3 * i + 1]], [a[3 * i + 2]], sb], [[b[3 * i]], [b[3 * i + 1]], [b[3 * i + 2]], db], p, q)
                      for i, (sb, db, p, q) in enumerate(s.reqs)]
        sizes = [t * block for t in toks]
        per_layer = sum(sizes) * pool
        s.src = _bytes(layers * per_layer, s.gen)
        s.dst = torch.zeros(layers * per_layer, dtype=torch.uint8, device=DEV)

        def tensors(flat):
            out = []
            for whole in _cut(flat, layers):
                at, ts = 0, []
                for size in sizes:
                    ts.append(whole[at:at + size * pool])
                    at += size * pool
                out.append(ts)
            return out

        _engine(s, tensors(s.src), tensors(s.dst), sizes, toks, shape, shape, PT.NVLINK, **kw)
        s.go = _submit
    if s.cli is not None:
        _open(s)
    return s


def _open(s: _State) -> None:
    """The peer has been talked to before: one step has gone over the channel (its bytes are taken back)."""
    s.go(s)
    s.dst.zero_()


def _prepare_store(s: _State) -> _State:
    c = s.case
    layers, n = c["layers"], c["blocks"]
    lay = AttnLayout(CacheShape.FLASH, n + n // 8 + 2, BLOCK, 8, DIM, 2)
    s.src = _normal_bf16(layers * lay.layer_bytes, s.gen)
    s.store_name = "perf_cases_%d_%d" % (os.getpid(), s.rng.getrandbits(48))
    s.store = PinnedKVStore(s.store_name, lay, _cut(s.src, layers), 0, 1, n, create=True, fp8=c["fp8"])
    keys = s.store.keys([s.rng.randrange(32000) for _ in range(n * BLOCK)], n)
    s.blocks, s.slots = s.rng.sample(range(1, lay.num_blocks), n), [slot for _, slot in s.store.reserve(keys)[0]]
    if c["load"]:
        s.store.save_layers(0, layers, s.blocks, s.slots).synchronize()
        s.store.seal(keys)
        s.src.zero_()
    else:
        s.store.host.zero_()
    return s


def run(state: _State):
    c = state.case
    if c["kind"] == "store":
        move = state.store.load_layers if c["load"] else state.store.save_layers
        # the caller seals (or uses) the blocks when the event says that they have arrived
        move(0, c["layers"], state.blocks, state.slots).synchronize()
        out = (state.src if c["load"] else state.store.host).view(torch.int64)
        out.owner = state           # the arena is unmapped with the store
        return out
    state.go(state)
    return state.dst.view(torch.int64)


def work(case: dict) -> dict:
    """Every byte of the moved rows (and pages of state) read once and written once; block tables are negligible."""
    kind, layers, tokens = case["kind"], case["layers"], case.get("tokens", 0)
    if kind in ("push", "fp8"):
        row = min(8 // case["p_tp"], 8 // case["d_tp"]) * 2 * DIM       # values of a token and layer, K and V
        per = row * 2 + (row + row // 32 if kind == "fp8" else row * 2)
    elif kind == "direct":
        row = case["heads"] * 2 * DIM
        per = row * 2 + (row * 2 if case["mode"] == MODE_COPY else row + row // 32)
    elif kind == "store":
        row = 8 * 2 * DIM
        tokens = case["blocks"] * BLOCK
        per = row * 2 + (row + row // 32 if case["fp8"] else row * 2)
    elif kind == "mla":
        per = 2 * sum(MLA_TOKEN)
    elif kind == "gdn":
        return {"bytes": 2 * layers * (tokens * GDN_TOKEN + min(case["reqs"], tokens) * 3 * GDN_STATE), "flops": 0}
    else:
        per = 2 * 8 * 2 * DIM * 2
    return {"bytes": per * tokens * layers, "flops": 0}


def tolerance(case: dict):
    """Copies are copies, the quantiser's codes and scales are defined bit by bit, and an e4m3 code times a power of two is a
    bf16 number: nothing may differ."""
    return "exact"
