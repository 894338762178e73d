"""Expert parallelism on GPUs: the expert-parallel layer against the oracle -- over peer memory (the C ABI's
shrike_ep_*) and over NCCL all-to-all (the checker) -- with one rank always, with two ranks when the box has
two GPUs; the pack kernel against the numpy protocol; the full-size mixed batch; and a wait that runs out
because nothing ever writes its word (a peer that never answers, made on the host)."""
import dataclasses
import os
import socket
import sys

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _free_port():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def _config(ne=16, act=None):
    from shrike_b200 import capi
    from shrike_b200.moe import MoEConfig
    return MoEConfig(d=256, f=128, num_experts=ne, top_k=4, act_dtype=capi.DTYPE_FP32 if act is None else act,
                     has_shared=True, shared_gated=False, shared_f=128, max_tokens=256)


def _problem(T, cfg, seed=5):
    import fixtures as fx
    rng = np.random.default_rng(seed)
    x = fx.round_bf16(rng.normal(0, 1, (T, cfg.d)).astype(np.float32))
    router = rng.normal(0, 0.05, (cfg.num_experts, cfg.d)).astype(np.float32)
    return x, router


def _oracle(cfg, x, router, seed):
    import oracle_lib as O
    import fixtures as fx
    T = x.shape[0]
    ids = np.zeros((T, cfg.top_k), np.uint32)
    w = np.zeros((T, cfg.top_k), np.float32)
    for t in range(T):
        ids[t], w[t] = O.router_select(O.router_logits_f32(router, x[t]), cfg.top_k, round_f16=True)
    ecfg = O.expert_cfg(cfg.d, cfg.f)
    blocks = {int(e): fx.synth_block(cfg, seed, 0, int(e)) for e in np.unique(ids)}
    shared = fx.synth_block(cfg, seed, 0, 100000, shared=True)
    y = O.moe_layer(O.layer_cfg(ecfg, O.expert_cfg(cfg.d, cfg.shared_f), False), blocks, shared, None, x, ids, w)
    return ids, w, y


def _build_layer(cfg, rank, world, per, seed, exchange, group=None):
    from shrike_b200 import capi
    import fixtures as fx
    from shrike_b200.ep import ExpertParallelLayer
    from shrike_b200.moe import expert_offsets
    layer = ExpertParallelLayer(cfg, rank, world, rank if torch.cuda.device_count() > rank else 0, per, group,
                                exchange=exchange)
    for e in range(layer.lo, layer.hi):
        layer.pool.upload(e - layer.lo, fx.synth_block(cfg, seed, 0, e))
    sh = torch.from_numpy(fx.synth_block(cfg, seed, 0, 100000, shared=True).copy()).to(layer.dev)
    layer._shared_block = sh
    layer.set_shared(capi.SharedExpert(sh.data_ptr(), expert_offsets(cfg, shared=True)[0]))
    return layer


def _run_rank(rank, world, port, T, seed, out_path, exchange="peer"):
    """One EP rank: builds its shard, runs the layer twice on its rows, saves y, hidden and the routing."""
    import torch.distributed as dist
    from shrike_b200.moe import RouterOperands
    cfg = _config()
    torch.cuda.set_device(rank)
    group = None
    if world > 1:
        os.environ["MASTER_ADDR"] = "127.0.0.1"
        os.environ["MASTER_PORT"] = str(port)
        os.environ.setdefault("NCCL_NVLS_ENABLE", "0")
        dist.init_process_group("nccl", rank=rank, world_size=world, device_id=torch.device("cuda", rank))
    x, router = _problem(T, cfg)
    per = T // world
    layer = _build_layer(cfg, rank, world, per, seed, exchange, group)
    dev = layer.dev
    ops = RouterOperands(weights=torch.from_numpy(router).to(dev))
    xl = torch.from_numpy(x[rank * per:(rank + 1) * per].copy()).to(dev)
    y = torch.empty_like(xl)
    h = xl.clone()
    for _ in range(2):  # a second pass reuses every buffer
        h.copy_(xl)
        layer.forward(ops, xl, y, h)
    layer.status()
    np.save(out_path, np.stack([y.cpu().numpy(), h.cpu().numpy()]))
    ids, _ = layer.routing(ops, xl)
    np.save(out_path + ".ids.npy", ids.cpu().numpy().astype(np.uint32))
    if exchange == "peer":
        sent, received, nbytes = layer.last_counts()
        np.save(out_path + ".counts.npy", np.array(sent + [received, nbytes], dtype=np.int64))
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    layer.close()


@pytest.mark.parametrize("exchange", ["peer", "nccl"])
@pytest.mark.parametrize("T", [8, 96])
def test_single_rank_expert_parallel_layer(cuda_device, tmp_path, T, exchange):
    seed = 21
    out = str(tmp_path / "y0.npy")
    _run_rank(0, 1, 0, T, seed, out, exchange)
    cfg = _config()
    x, router = _problem(T, cfg)
    ids, w, y_ref = _oracle(cfg, x, router, seed)
    got = np.load(out)
    assert (np.load(out + ".ids.npy") == ids).all()
    assert np.linalg.norm(got[0] - y_ref) / np.linalg.norm(y_ref) <= 1e-3
    assert np.abs(got[1] - (x + got[0])).max() <= 1e-5 * np.abs(x).max()
    if exchange == "peer":
        counts = np.load(out + ".counts.npy")
        assert counts[0] == T and counts[1] == T   # every row has a pick on the only rank; nothing leaves it
        assert counts[2] == 0


def _edges(call):
    """(all, programmatic) edges of the graph that the call's launches make on a stream of their own."""
    import ctypes as C
    rt = C.CDLL("libcudart.so.12")
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    graph, n = C.c_void_p(), C.c_size_t()
    with torch.cuda.stream(stream):
        assert rt.cudaStreamBeginCapture(C.c_void_p(stream.cuda_stream), 1) == 0   # 1: this thread's calls
        try:
            call()
        finally:
            assert rt.cudaStreamEndCapture(C.c_void_p(stream.cuda_stream), C.byref(graph)) == 0
    assert rt.cudaGraphGetEdges_v2(graph, None, None, None, C.byref(n)) == 0
    ends, data = (C.c_void_p * n.value), (C.c_uint8 * 8 * n.value)()
    assert rt.cudaGraphGetEdges_v2(graph, ends(), ends(), data, C.byref(n)) == 0
    assert rt.cudaGraphDestroy(graph) == 0
    return n.value, sum(e[2] == 1 for e in data)   # cudaGraphEdgeData.type, cudaGraphDependencyTypeProgrammatic


def test_handles_launch_as_before_once_a_forward_is_over(cuda_device):
    """An expert-parallel forward launches its kernels without overlap of successive ones; the handles' own prefill
    calls have it before the layer is made, after a forward, and after the layer has gone."""
    from shrike_b200.moe import RouterOperands
    cfg, T = _config(), 96
    layer = _build_layer(cfg, 0, 1, T, 3, "peer")
    x_np, router = _problem(T, cfg)
    ops = RouterOperands(weights=torch.from_numpy(router).cuda())
    x = torch.from_numpy(x_np).cuda()
    y = torch.empty_like(x)
    ids, w = torch.zeros((T, cfg.top_k), dtype=torch.int32, device="cuda"), torch.zeros((T, cfg.top_k), device="cuda")
    layer.home.encode_router(ops, x, ids, w)
    slots = torch.full_like(ids, -1)

    def prefill():
        layer.home.encode_prefill(layer.pool, layer.offsets, ids, slots, w, x, y, None, layer.shared)

    prefill()
    before = _edges(prefill)
    layer.forward(ops, x, y)
    layer.status()
    assert before[1] > 0 and _edges(prefill) == before
    layer._lib.shrike_ep_destroy(layer._ep)
    layer._ep = None
    assert _edges(prefill) == before
    layer.close()


def test_what_creation_clears_is_clear_when_it_returns(cuda_device):
    """Handles, residency tables and exchange buffers are cleared on the legacy stream, which a caller's non-blocking
    stream does not wait for: every create call waits itself, behind whatever that stream still has to do (20 ms here)."""
    import ctypes as C
    from shrike_b200 import capi
    from shrike_b200.ep import ExpertParallelLayer
    from shrike_b200.moe import MoE
    cfg = _config()
    legacy = torch.cuda.default_stream()
    layer = ExpertParallelLayer(cfg, 0, 1, 0, 96)
    lib, made = capi.load(), C.c_void_p()

    def after(create):
        torch.cuda._sleep(40_000_000)
        assert not legacy.query()
        create()
        assert legacy.query()

    moes = []
    after(lambda: moes.append(MoE(cfg)))
    after(lambda: moes[0].create_residency(1))
    after(lambda: layer.home._check(lib.shrike_ep_create(layer.home._h, layer.routed._h, 0, 1, 96, C.byref(made))))
    lib.shrike_ep_destroy(made)
    moes[0].close()
    layer.close()


def test_cuda_dispatch_matches_the_protocol(cuda_device):
    import ep_reference as R
    T, seed = 96, 22
    cfg = _config()
    x, router = _problem(T, cfg)
    ids, w, _ = _oracle(cfg, x, router, seed)
    # the rows packed for an imagined 4-rank world, through the C ABI
    from shrike_b200.moe import MoE, _ptr, _stream
    moe = MoE(dataclasses.replace(cfg, max_tokens=T))
    dev = torch.device("cuda:0")
    world, epr, cap = 4, cfg.num_experts // 4, T
    xd = torch.from_numpy(x).to(dev)
    idd = torch.from_numpy(ids.astype(np.int32)).to(dev)
    wd = torch.from_numpy(w).to(dev)
    sx = torch.zeros((world, cap, cfg.d), dtype=torch.float32, device=dev)
    si = torch.zeros((world, cap, cfg.top_k), dtype=torch.int32, device=dev)
    sw = torch.zeros((world, cap, cfg.top_k), dtype=torch.float32, device=dev)
    sc = torch.zeros(world, dtype=torch.int32, device=dev)
    ro = torch.zeros((T, world), dtype=torch.int32, device=dev)
    moe._check(moe._lib.shrike_ep_encode_dispatch(moe._h, _stream(), _ptr(xd), _ptr(idd), _ptr(wd), T, world, epr, cap,
                                                  _ptr(sx), _ptr(si), _ptr(sw), _ptr(sc), _ptr(ro)))
    moe.status()
    rx, ri, rw, rc, rr = R.pack(x, ids, w, world, epr, cap)
    assert (sc.cpu().numpy() == rc).all() and (ro.cpu().numpy() == rr).all()
    assert (si.cpu().numpy().astype(np.uint32) == ri).all()
    for g in range(world):
        n = int(rc[g])
        assert (sx.cpu().numpy()[g, :n] == rx[g, :n]).all() and (sw.cpu().numpy()[g, :n] == rw[g, :n]).all()
    moe.close()


def test_full_size_mixed_batch_on_one_rank(cuda_device):
    """The expert-parallel workload at its full per-rank size: 16 decode rows + one 2048-row prefill chunk of the
    Kimi-Linear shape (int8 g64, 256 experts top-8 sigmoid with a selection bias, shared expert), bf16 rows in,
    fp32 rows out, through the peer-memory layer with every expert on this rank; sampled rows against the oracle."""
    import fixtures as fx
    import oracle_lib as O
    from shrike_b200 import capi
    from shrike_b200.ep import ExpertParallelLayer
    from shrike_b200.moe import RouterOperands, expert_offsets
    from gpu_harness import bf16_tensor
    rows, seed = 16 + 2048, 31
    cfg = fx.kimi_config(max_tokens=rows)
    dev = torch.device("cuda:0")
    layer = ExpertParallelLayer(cfg, 0, 1, 0, rows)
    layer.pool.fill_synthetic(0, layer.epr, seed, 0, first_expert=0)
    soff, _ = expert_offsets(cfg, shared=True)
    sh = torch.from_numpy(fx.synth_block(cfg, seed, 0, 100000, shared=True).copy()).to(dev)
    layer.set_shared(capi.SharedExpert(sh.data_ptr(), soff))
    rng = np.random.default_rng(seed)
    router = rng.normal(0, 0.05, (cfg.num_experts, cfg.d)).astype(np.float32)
    correction = rng.uniform(-0.1, 0.1, cfg.num_experts).astype(np.float32)
    xr = fx.round_bf16(rng.normal(0, 1, (rows, cfg.d)).astype(np.float32))
    ops = RouterOperands(weights=torch.from_numpy(router).to(dev), logit_bias=bf16_tensor(correction, dev))
    x = torch.from_numpy(xr).to(torch.bfloat16).to(dev)
    y = torch.empty((rows, cfg.d), dtype=torch.float32, device=dev)
    layer.forward(ops, x, y)
    layer.status()
    ids, w = layer.routing(ops, x)
    ids, w = ids.cpu().numpy().astype(np.uint32), w.cpu().numpy()
    assert all(len(set(r)) == cfg.top_k for r in ids[:64].tolist())
    sample = np.sort(rng.choice(rows, 40, replace=False))
    ecfg = O.expert_cfg(cfg.d, cfg.f, bits=8)
    lcfg = O.layer_cfg(ecfg, O.expert_cfg(cfg.d, cfg.shared_f, bits=8), False)
    blocks = {int(e): fx.synth_block(cfg, seed, 0, int(e)) for e in np.unique(ids[sample])}
    ref = O.moe_layer(lcfg, blocks, fx.synth_block(cfg, seed, 0, 100000, shared=True), None, xr[sample], ids[sample],
                      w[sample], threads=os.cpu_count() or 8)
    got = y.cpu().numpy()[sample]
    assert np.isfinite(y.cpu().numpy()).all()
    assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= 1e-3
    sent, received, nbytes = layer.last_counts()
    assert sent[0] == rows and received == rows and nbytes == 0
    layer.close()


def test_a_peer_that_never_answers_ends_in_a_timeout_status(cuda_device):
    """Rank 0 of an imagined two-rank world whose peer buffer is plain memory that nothing writes: the bounded
    waits for the peer's arrival words run out, the call returns, and the status says timeout. No GPU fault, no
    second process: the failure is made on the host by never starting the peer."""
    from shrike_b200 import capi
    from shrike_b200.ep import ExpertParallelLayer
    from shrike_b200.moe import RouterOperands, ShrikeError, expert_offsets
    cfg = _config()
    T, seed = 32, 24
    x, router = _problem(T, cfg)
    dev = torch.device("cuda:0")
    layer = ExpertParallelLayer(cfg, 0, 2, 0, T, None, exchange="peer", connect=False)
    base, nbytes = layer.buffer()
    fake_peer = torch.zeros(nbytes, dtype=torch.uint8, device=dev)   # the peer that never runs
    layer.connect_pointers([base, fake_peer.data_ptr()])
    layer.set_wait_polls(200)   # a fraction of a millisecond per wait
    import fixtures as fx
    for e in range(layer.lo, layer.hi):
        layer.pool.upload(e - layer.lo, fx.synth_block(cfg, seed, 0, e))
    sh = torch.from_numpy(fx.synth_block(cfg, seed, 0, 100000, shared=True).copy()).to(dev)
    layer.set_shared(capi.SharedExpert(sh.data_ptr(), expert_offsets(cfg, shared=True)[0]))
    ops = RouterOperands(weights=torch.from_numpy(router).to(dev))
    xd = torch.from_numpy(x).to(dev)
    y = torch.empty_like(xd)
    layer.forward(ops, xd, y)   # returns: every wait is bounded
    with pytest.raises(ShrikeError) as err:
        layer.status()
    assert err.value.code == capi.ETIMEDOUT
    assert torch.isfinite(y).all()
    # the context is intact: a one-rank layer on the same GPU still answers
    torch.cuda.synchronize()
    layer.close()
    out_ok = torch.zeros(4, device=dev) + 1
    assert float(out_ok.sum()) == 4.0


def _two_ranks(tmp_path, exchange, T=96, seed=23):
    import subprocess
    world = 2
    port = _free_port()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    procs = []
    for r in range(world):
        code = (f"import sys; sys.path.insert(0, {root!r}); sys.path.insert(0, {root + '/tests'!r}); "
                f"import test_gpu_ep as t; t._run_rank({r}, {world}, {port}, {T}, {seed}, "
                f"{str(tmp_path / f'y{r}.npy')!r}, {exchange!r})")
        procs.append(subprocess.Popen([sys.executable, "-c", code]))
    for p in procs:
        assert p.wait(timeout=300) == 0
    cfg = _config()
    x, router = _problem(T, cfg)
    ids, w, y_ref = _oracle(cfg, x, router, seed)
    y = np.concatenate([np.load(str(tmp_path / f"y{r}.npy"))[0] for r in range(world)])
    assert np.linalg.norm(y - y_ref) / np.linalg.norm(y_ref) <= 1e-3
    return ids


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_two_ranks_over_peer_memory_match_the_oracle(cuda_device, tmp_path):
    ids = _two_ranks(tmp_path, "peer")
    # rows sent: rank r's rows with a pick in each half of the experts
    cfg = _config()
    per = ids.shape[0] // 2
    for r in range(2):
        counts = np.load(str(tmp_path / f"y{r}.npy.counts.npy"))
        mine = ids[r * per:(r + 1) * per]
        for g in range(2):
            assert counts[g] == int(((mine // (cfg.num_experts // 2)) == g).any(axis=1).sum())


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_two_nccl_ranks_match_the_oracle(cuda_device, tmp_path):
    _two_ranks(tmp_path, "nccl")


@pytest.mark.parametrize("T", [8, 96])
def test_int8_shared_expert_beside_int4_routed_experts(cuda_device, T):
    """The reference's Qwen layers keep the shared expert in int8 and the routed experts in int4
    (SharedExpertInt8.swift:55-227): the home handle describes the shared expert's block, the routed handle the
    routed experts'; one rank. Against the oracle with the two formats."""
    import fixtures as fx
    import oracle_lib as O
    from shrike_b200 import capi
    from shrike_b200.ep import ExpertParallelLayer
    from shrike_b200.moe import RouterOperands, expert_offsets
    seed = 27
    cfg4 = _config()                                         # routed experts: int4
    cfg8 = dataclasses.replace(cfg4, weight_bits=8)          # the shared expert's format
    x, router = _problem(T, cfg4)
    dev = torch.device("cuda:0")
    layer = ExpertParallelLayer(cfg8, 0, 1, 0, T, None, exchange="peer", routed_config=cfg4)
    for e in range(layer.lo, layer.hi):
        layer.pool.upload(e - layer.lo, fx.synth_block(cfg4, seed, 0, e))
    sh_block = fx.synth_block(cfg8, seed, 0, 100000, shared=True)
    sh = torch.from_numpy(sh_block.copy()).to(dev)
    layer.set_shared(capi.SharedExpert(sh.data_ptr(), expert_offsets(cfg8, shared=True)[0]))
    ops = RouterOperands(weights=torch.from_numpy(router).to(dev))
    xd = torch.from_numpy(x).to(dev)
    y = torch.empty_like(xd)
    layer.forward(ops, xd, y)
    layer.status()
    ids = np.zeros((T, cfg4.top_k), np.uint32)
    w = np.zeros((T, cfg4.top_k), np.float32)
    for t in range(T):
        ids[t], w[t] = O.router_select(O.router_logits_f32(router, x[t]), cfg4.top_k, round_f16=True)
    blocks = {int(e): fx.synth_block(cfg4, seed, 0, int(e)) for e in np.unique(ids)}
    lcfg = O.layer_cfg(O.expert_cfg(cfg4.d, cfg4.f), O.expert_cfg(cfg4.d, cfg4.shared_f, bits=8), False)
    y_ref = O.moe_layer(lcfg, blocks, sh_block, None, x, ids, w)
    got = y.cpu().numpy()
    assert np.linalg.norm(got - y_ref) / np.linalg.norm(y_ref) <= 1e-3
    layer.close()


@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
def test_output_rows_that_are_not_whole_vectors(cuda_device, dtype):
    """y and hidden one element into a buffer: combined by single elements, with the results of aligned rows. (The down
    projection's sums are added in no fixed order: two units of the last place.)"""
    from shrike_b200 import capi
    from shrike_b200.moe import RouterOperands
    cfg = _config(act=capi.DTYPE_FP32 if dtype == "fp32" else capi.DTYPE_BF16)
    x, router = _problem(40, cfg)
    layer = _build_layer(cfg, 0, 1, 40, 9, "peer")
    ops = RouterOperands(weights=torch.from_numpy(router).to(layer.dev))
    xl = torch.from_numpy(x).to(layer.dev).to(cfg.torch_act_dtype)
    got = []
    for skip in (0, 1):
        y = torch.zeros(xl.numel() + 8, dtype=cfg.torch_y_dtype, device=layer.dev)[skip:skip + xl.numel()].view(xl.shape)
        h = torch.zeros(xl.numel() + 8, dtype=xl.dtype, device=layer.dev)[skip:skip + xl.numel()].view(xl.shape).copy_(xl)
        layer.forward(ops, xl, y, h)
        layer.status()
        got.append((y.float(), h.float()))
    layer.close()
    ulp = 2.0 ** (-22 if dtype == "fp32" else -7)
    assert not torch.equal(got[0][0], torch.zeros_like(got[0][0]))
    for a, b in zip(*got):
        assert ((a - b).abs() <= 2 * ulp * a.abs() + 1e-6 * a.abs().max()).all()


def _view(address, nbytes):
    """The device memory at an address, as a byte tensor over it."""
    class Memory:
        __cuda_array_interface__ = dict(shape=(nbytes,), typestr="|u1", data=(address, False), version=3)
    return torch.as_tensor(Memory(), device="cuda")


def _exchange_areas(cfg, world, cap, buf):
    """A rank's exchange buffer by its areas, each a multiple of 256 bytes: rows, ids and weights received from every rank,
    partial rows returned, and the two arrival words."""
    at, areas = 0, []
    for shape, dtype in (((world, cap, cfg.d), cfg.torch_act_dtype), ((world, cap, cfg.top_k), torch.int32),
                         ((world, cap, cfg.top_k), torch.float32), ((world, cap, cfg.d), cfg.torch_y_dtype),
                         ((world,), torch.int64), ((world,), torch.int64)):
        n = int(np.prod(shape)) * torch.empty((), dtype=dtype).element_size()
        areas.append(buf[at:at + n].view(dtype).view(shape))
        at = (at + n + 255) // 256 * 256
    assert at == buf.numel()
    return areas


@pytest.mark.parametrize("T,dtype", [(1, "fp32"), (37, "fp32"), (37, "bf16"), (90, "bf16")])
def test_both_ranks_rows_beside_words_that_are_there(cuda_device, T, dtype):
    """Rank 0 of a two-rank world, and rank 1 made on the host: before the call its rows, its partial rows and both of its
    arrival words are in rank 0's buffer, so no wait waits. Rank 0's y are its own picks, the returned rows and the shared
    expert; what it sends and returns is in rank 1's buffer, and nothing in its own return area."""
    import ep_reference as R
    import fixtures as fx
    import oracle_lib as O
    from shrike_b200 import capi
    from shrike_b200.ep import ExpertParallelLayer
    from shrike_b200.moe import RouterOperands, expert_offsets
    cfg, seed, world = _config(act=capi.DTYPE_FP32 if dtype == "fp32" else capi.DTYPE_BF16), 26, 2
    x, router = _problem(world * T, cfg)
    ids, w, y_ref = _oracle(cfg, x, router, seed)
    layer = ExpertParallelLayer(cfg, 0, world, 0, T, None, exchange="peer", connect=False)
    epr = layer.epr
    for e in range(layer.lo, layer.hi):
        layer.pool.upload(e - layer.lo, fx.synth_block(cfg, seed, 0, e))
    sh = torch.from_numpy(fx.synth_block(cfg, seed, 0, 100000, shared=True).copy()).cuda()
    layer.set_shared(capi.SharedExpert(sh.data_ptr(), expert_offsets(cfg, shared=True)[0]))
    base, nbytes = layer.buffer()
    peer = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    layer.connect_pointers([base, peer.data_ptr()])
    mine, theirs = _exchange_areas(cfg, world, T, _view(base, nbytes)), _exchange_areas(cfg, world, T, peer)
    blocks = {e: fx.synth_block(cfg, seed, 0, e) for e in range(cfg.num_experts)}
    lcfg = O.layer_cfg(O.expert_cfg(cfg.d, cfg.f), None, False)

    def partial(rank, rows):   # the rows' picks on a rank, added in fp32
        return O.moe_layer(lcfg, blocks, None, None, x[rows], ids[rows], np.where(ids[rows] // epr == rank, w[rows], np.float32(0)))

    home, away = np.arange(T), np.arange(T, 2 * T)   # rank 0's rows, rank 1's
    sent, back = R.pack(x[home], ids[home], w[home], world, epr, T), R.pack(x[away], ids[away], w[away], world, epr, T)
    on_1, from_1 = (ids[home] // epr == 1).any(axis=1), (ids[away] // epr == 0).any(axis=1)
    ops = RouterOperands(weights=torch.from_numpy(router).cuda())
    xd = torch.from_numpy(x[home]).cuda().to(cfg.torch_act_dtype)
    y, h = torch.empty((T, cfg.d), dtype=cfg.torch_y_dtype, device="cuda"), torch.empty_like(xd)
    tol = 1e-3 if dtype == "fp32" else 1e-3 + 3 * 2.0 ** -9   # bf16: both partial rows and their sum are rounded
    for call in (1, 2):
        mine[0][1, :from_1.sum()] = torch.from_numpy(back[0][0, :from_1.sum()]).cuda().to(cfg.torch_act_dtype)
        mine[1][1] = torch.from_numpy(back[1][0].view(np.int32)).cuda()
        mine[2][1] = torch.from_numpy(back[2][0]).cuda()
        mine[3].fill_(7.0)
        mine[3][1, :on_1.sum()] = torch.from_numpy(partial(1, home[on_1])).cuda().to(cfg.torch_y_dtype)
        mine[4][1] = call << 32 | int(from_1.sum())
        mine[5][1] = call << 32
        theirs[3].fill_(-7.0)
        h.copy_(xd)
        torch.cuda.synchronize()
        layer.forward(ops, xd, y, h)
        layer.status()
        got = y.float().cpu().numpy()
        assert np.linalg.norm(got - y_ref[home]) <= tol * np.linalg.norm(y_ref[home])
        assert torch.equal(h, (xd.float() + y.float()).to(h.dtype))
        n = int(sent[3][1])
        assert int(theirs[4][0]) == call << 32 | n and int(theirs[5][0]) == call << 32
        assert torch.equal(theirs[0][0, :n].float().cpu(), torch.from_numpy(sent[0][1, :n]))
        assert (theirs[1][0, :n].cpu().numpy().view(np.uint32) == sent[1][1, :n]).all()
        assert (theirs[2][0, :n].cpu().numpy() == sent[2][1, :n]).all()
        n = int(from_1.sum())
        want = partial(0, away[from_1])
        assert np.linalg.norm(theirs[3][0, :n].float().cpu().numpy() - want) <= tol * np.linalg.norm(want)
        assert (theirs[3][0, n:] == -7.0).all() and (theirs[3][1] == -7.0).all() and (mine[3][0] == 7.0).all()
        assert layer.last_counts()[0] == [int(sent[3][0]), int(sent[3][1])] and layer.last_counts()[1] == int(sent[3][0]) + n
    layer.close()


@pytest.mark.parametrize("T,world,skip", [(1, 1, 0), (5, 3, 1), (37, 8, 0), (65536 + 37, 2, 0), (65536 + 3, 2, 1)])
def test_combine_matches_the_protocol(cuda_device, T, world, skip):
    """More rows than one launch numbers, ranks in whole and broken fours, rows that are not whole vectors: the sums in rank order."""
    import ep_reference as R
    from shrike_b200.moe import MoE, _ptr, _stream
    cfg = dataclasses.replace(_config(), d=64)
    moe = MoE(cfg)
    rng = np.random.default_rng(T)
    cap = min(T, 300)
    recv = rng.normal(0, 1, (world, cap, 64)).astype(np.float32)
    row_of = rng.integers(-1, cap, (T, world)).astype(np.int32)
    home, x = rng.normal(0, 1, (T, 64)).astype(np.float32), rng.normal(0, 1, (T, 64)).astype(np.float32)
    y, h = (torch.zeros(T * 64 + 8, device="cuda")[skip:skip + T * 64].view(T, 64) for _ in range(2))
    h.copy_(torch.from_numpy(x))
    operands = [torch.from_numpy(v).cuda() for v in (recv, row_of, home)]   # (held until the call is over)
    moe._check(moe._lib.shrike_ep_encode_combine(moe._h, _stream(), *map(_ptr, operands), T, world, cap, _ptr(y), _ptr(h)))
    moe.status()
    want = home.copy()
    for g in range(world):
        want += np.where(row_of[:, g, None] >= 0, recv[g][np.maximum(row_of[:, g], 0)], np.float32(0))
    if T < 100:
        assert np.array_equal(want, R.combine(recv, row_of, home))
    assert (y.cpu().numpy() == want).all() and (h.cpu().numpy() == x + want).all()
    moe.close()


@pytest.mark.parametrize("T", [1, 2, 64, 65, 200])
@pytest.mark.parametrize("shared", [True, False])
def test_a_rank_alone_gives_what_the_exchange_gives(cuda_device, T, shared):
    """A world of one runs the home handle's layer call; rows whose y begins inside x take the general way through the exchange
    buffer. Both against the oracle, the residual and the counters."""
    from shrike_b200.moe import RouterOperands
    seed = 31
    cfg = dataclasses.replace(_config(), **({} if shared else dict(has_shared=False, shared_f=0)))
    x, router = _problem(T, cfg)
    ids, w, y_ref = _oracle(_config(), x, router, seed)
    if not shared:
        import fixtures as fx
        import oracle_lib as O
        ecfg = O.expert_cfg(cfg.d, cfg.f)
        y_ref = O.moe_layer(O.layer_cfg(ecfg, None, False), {int(e): fx.synth_block(cfg, seed, 0, int(e)) for e in np.unique(ids)}, None, None,
                            x, ids, w)
    layer = _build_alone(cfg, T, seed)
    ops = RouterOperands(weights=torch.from_numpy(router).to(layer.dev))
    for across in (False, True):
        buf = torch.zeros((2 * T + 1, cfg.d), device=layer.dev)
        xd, y = buf[:T], buf[1:T + 1] if across else buf[T:2 * T]
        xd.copy_(torch.from_numpy(x))
        h = torch.from_numpy(x).to(layer.dev)
        layer.forward(ops, xd, y, h)
        layer.status()
        got = y.cpu().numpy()
        assert np.linalg.norm(got - y_ref) / np.linalg.norm(y_ref) <= 1e-3
        assert np.abs(h.cpu().numpy() - (x + got)).max() <= 1e-5 * np.abs(x).max()
        assert layer.last_counts() == ([T], T, 0)
    layer.close()


def _build_alone(cfg, T, seed):
    import fixtures as fx
    from shrike_b200.ep import ExpertParallelLayer
    if cfg.has_shared:
        return _build_layer(cfg, 0, 1, T, seed, "peer")
    layer = ExpertParallelLayer(cfg, 0, 1, 0, T)
    for e in range(layer.lo, layer.hi):
        layer.pool.upload(e, fx.synth_block(cfg, seed, 0, e))
    return layer


def test_a_replayed_forward_counts_its_own_rows(cuda_device):
    from shrike_b200.moe import RouterOperands
    cfg = _config()
    x, router = _problem(8, cfg)
    layer = _build_layer(cfg, 0, 1, 8, 32, "peer")
    ops = RouterOperands(weights=torch.from_numpy(router).to(layer.dev))
    xd = torch.from_numpy(x).to(layer.dev)
    y, y4 = torch.zeros_like(xd), torch.zeros_like(xd[:4])
    layer.forward(ops, xd, y)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.forward(ops, xd, y)
    want = y.clone()
    layer.forward(ops, xd[:4], y4)
    torch.cuda.synchronize()
    assert layer.last_counts()[:2] == ([4], 4)
    y.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert layer.last_counts()[:2] == ([8], 8) and torch.equal(y, want)
    layer.close()


def _exchanges(layer):
    """Forwards that went through the exchange buffer: the epoch of this rank's arrival word for itself."""
    torch.cuda.synchronize()
    return int(_exchange_areas(layer.cfg, layer.world, layer.cap, _view(*layer.buffer()))[4][layer.rank]) >> 32


def _rows(cfg, x, across, skip=0):
    """x, and y: rows of their own, or beginning 16 bytes into x, `skip` elements further on."""
    esz = torch.empty((), dtype=cfg.torch_y_dtype).element_size()
    n_x, n_y = x.numel() * x.element_size(), x.numel() * esz
    buf = torch.zeros(n_x + n_y + 64, dtype=torch.uint8, device=x.device)
    at = (16 if across else (n_x + 15) // 16 * 16) + skip * esz
    xd, y = buf[:n_x].view(x.dtype).view(x.shape), buf[at:at + n_y].view(cfg.torch_y_dtype).view(x.shape)
    return xd.copy_(x), y


@pytest.fixture
def exchanged(monkeypatch):
    """A world of one exchanges with itself where its layer call does not take the rows: every forward's y begins inside x
    here, as far from a whole 16 bytes as the test's own."""
    from shrike_b200.ep import ExpertParallelLayer
    inner = ExpertParallelLayer.forward

    def forward(self, router, x, y, hidden=None):
        xd, yd = _rows(self.cfg, x, True, y.data_ptr() % 16 // y.element_size())
        before = _exchanges(self)
        inner(self, router, xd, yd, hidden)
        y.copy_(yd)
        assert _exchanges(self) == before + 1
    monkeypatch.setattr(ExpertParallelLayer, "forward", forward)
    return inner


@pytest.mark.parametrize("T", [8, 96])
def test_single_rank_through_the_exchange_buffer(cuda_device, tmp_path, exchanged, T):
    test_single_rank_expert_parallel_layer(cuda_device, tmp_path, T, "peer")


def test_full_size_mixed_batch_through_the_exchange_buffer(cuda_device, exchanged):
    test_full_size_mixed_batch_on_one_rank(cuda_device)


@pytest.mark.parametrize("dtype", ["fp32", "bf16"])
def test_exchanged_output_rows_that_are_not_whole_vectors(cuda_device, exchanged, dtype):
    test_output_rows_that_are_not_whole_vectors(cuda_device, dtype)


def test_handles_launch_as_before_once_rows_were_exchanged(cuda_device, exchanged):
    """The forward that exchanges sets the handles' launches itself, and puts them back."""
    from shrike_b200.moe import RouterOperands
    test_handles_launch_as_before_once_a_forward_is_over(cuda_device)
    cfg, T = _config(), 96
    layer = _build_layer(cfg, 0, 1, T, 3, "peer")
    x, router = _problem(T, cfg)
    xd, y = _rows(cfg, torch.from_numpy(x).cuda(), True)
    ops = RouterOperands(weights=torch.from_numpy(router).cuda())
    edges = _edges(lambda: exchanged(layer, ops, xd, y))   # (looked at, never run)
    assert edges[0] > 0 and edges[1] == 0
    layer.close()


@pytest.mark.parametrize("T", [1, 2, 64, 65, 200])
def test_which_rows_a_rank_alone_exchanges(cuda_device, T):
    """Those whose y begins inside x, and one row whose y or hidden is not 16-byte aligned; the same rows either way."""
    from shrike_b200.moe import RouterOperands
    cfg = _config()
    x, router = _problem(T, cfg)
    _, _, y_ref = _oracle(cfg, x, router, 31)
    layer = _build_layer(cfg, 0, 1, T, 31, "peer")
    ops = RouterOperands(weights=torch.from_numpy(router).to(layer.dev))
    exchanges = 0
    for across, skip_y, skip_h in ((False, 0, 0), (True, 0, 0), (False, 1, 0), (False, 0, 1)):
        xd, y = _rows(cfg, torch.from_numpy(x).to(layer.dev), across, skip_y)
        h = torch.zeros(x.size + 8, device=layer.dev)[skip_h:skip_h + x.size].view(x.shape)
        h.copy_(torch.from_numpy(x))
        layer.forward(ops, xd, y, h)
        layer.status()
        exchanges += across or (T == 1 and skip_y + skip_h > 0)
        assert _exchanges(layer) == exchanges
        got = y.cpu().numpy()
        assert np.linalg.norm(got - y_ref) / np.linalg.norm(y_ref) <= 1e-3
        assert np.abs(h.cpu().numpy() - (x + got)).max() <= 1e-5 * np.abs(x).max()
        assert layer.last_counts() == ([T], T, 0)
    layer.close()


@pytest.mark.parametrize("bits,act,f,T,exchanges", [
    (4, "silu", 192, 2, 0), (4, "silu", 192, 48, 0), (4, "silu", 192, 49, 1), (4, "silu", 192, 64, 1), (4, "silu", 128, 64, 0),
    (4, "clamped", 192, 1, 1), (4, "clamped", 192, 48, 1), (4, "clamped", 128, 5, 1), (8, "silu", 192, 64, 0), (8, "clamped", 192, 5, 0)])
def test_which_calls_of_nibbles_exchange(cuda_device, bits, act, f, T, exchanges):
    """A rank alone, a home handle of up to 64 rows. Where per-tile kernels would run the layer call (f 192: an odd number of groups) more than
    48 rows of nibbles go through the exchange, behind a clamped SwiGLU in groups of 64 all of them."""
    from gpu_harness import oracle_expert_cfg
    from shrike_b200 import capi
    from shrike_b200.moe import RouterOperands
    import fixtures as fx
    import oracle_lib as O
    cfg = dataclasses.replace(_config(), f=f, shared_f=f, weight_bits=bits, activation=capi.ACT_SILU if act == "silu" else capi.ACT_CLAMPED_SWIGLU)
    x, router = _problem(T, cfg)
    ids, w, _ = _oracle(_config(), x, router, 33)
    y_ref = O.moe_layer(O.layer_cfg(oracle_expert_cfg(cfg), oracle_expert_cfg(cfg, shared=True), False),
                        {int(e): fx.synth_block(cfg, 33, 0, int(e)) for e in np.unique(ids)}, fx.synth_block(cfg, 33, 0, 100000, shared=True), None, x, ids, w)
    layer = _build_layer(cfg, 0, 1, 64, 33, "peer")
    xd, y = _rows(cfg, torch.from_numpy(x).to(layer.dev), False)
    layer.forward(RouterOperands(weights=torch.from_numpy(router).to(layer.dev)), xd, y)
    layer.status()
    assert _exchanges(layer) == exchanges
    assert np.linalg.norm(y.cpu().numpy() - y_ref) / np.linalg.norm(y_ref) <= 1e-3
    assert layer.last_counts() == ([T], T, 0)
    layer.close()


@pytest.mark.parametrize("group,T", [(64, 1), (64, 5), (32, 1), (32, 5)])
def test_a_rank_alone_is_as_exact_as_the_exchange(cuda_device, group, T):
    """Large int4 experts with biases, an odd (groups of 64) and an even number of groups: against the oracle the rows of a call are
    at most half as much again as far off as those that go through the exchange buffer."""
    from gpu_harness import oracle_expert_cfg
    from shrike_b200 import capi
    from shrike_b200.moe import RouterOperands
    import fixtures as fx
    import oracle_lib as O
    cfg = dataclasses.replace(_config(8), d=2880, f=2880, group_size=group, top_k=2, activation=capi.ACT_CLAMPED_SWIGLU, expert_bias=True,
                              has_shared=False, shared_f=0)
    x, router = _problem(T, cfg)
    layer = _build_alone(cfg, T, 34)
    ops = RouterOperands(weights=torch.from_numpy(router).to(layer.dev))
    ids, w = (t.cpu().numpy() for t in layer.routing(ops, torch.from_numpy(x).to(layer.dev)))
    y_ref = O.moe_layer(O.layer_cfg(oracle_expert_cfg(cfg), None, False), {int(e): fx.synth_block(cfg, 34, 0, int(e)) for e in np.unique(ids)},
                        None, None, x, ids.astype(np.uint32), w)
    off = []
    for across in (False, True):
        xd, y = _rows(cfg, torch.from_numpy(x).to(layer.dev), across)
        layer.forward(ops, xd, y)
        layer.status()
        off.append(np.linalg.norm(y.cpu().numpy() - y_ref) / np.linalg.norm(y_ref))
    layer.close()
    assert off[1] <= 1e-3 and off[0] <= 1.5 * off[1], off
