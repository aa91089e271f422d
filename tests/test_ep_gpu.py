"""Expert-parallel MoE block of the runtime (ainfer_ep_*: batched router, device permute, grouped
tensor-core expert GEMMs, un-permute, slot-ordered combine; NCCL send/recv between ranks) against
the CPU oracle's single-token MoE block: every row of the batch bit for bit, with one rank and,
when two GPUs are visible, with two NCCL ranks that each hold half of the experts."""
import os
import socket

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def _oracle_rows(preset, seed, layer, res):
    """x[t] = res[t] + MoE(rmsnorm(res[t])) and the routed experts, by the oracle, per row."""
    import json
    cfg = json.loads(O.preset_json(preset))
    H, k = cfg["hidden"], cfg["top_k"]
    om = O.Model(arch_json=O.preset_json(preset), synth_seed=seed)
    pfx = f"model.language_model.layers.{layer}."
    w = O.bf16_to_f32(om.tensor(pfx + "post_attention_layernorm.weight")["data"].view(np.uint16))
    out = np.zeros_like(res)
    routed = np.zeros((res.shape[0], k), np.int32)
    for t in range(res.shape[0]):
        hn, y, gap = np.zeros(H, np.float32), np.zeros(H, np.float32), np.zeros(1, np.float32)
        O.lib().orc_rmsnorm(np.ascontiguousarray(res[t]), np.ascontiguousarray(w), H, float(cfg["rms_eps"]), hn)
        O.lib().orc_moe_block(om.h, pfx.encode(), hn, y, routed[t], gap)
        out[t] = res[t] + y
    om.close()
    return out, routed


def _batch(H, n, seed=5):
    return np.random.default_rng(seed).standard_normal((n, H)).astype(np.float32)


@pytest.mark.parametrize("preset,batch,layer", [("mini", 8, 1), ("mini", 64, 0), ("tiny", 3, 1), ("small", 64, 2)])
def test_one_rank_equals_oracle(preset, batch, layer):
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, f"synth:{preset}:seed=2")
    H, k = model.config["hidden"], model.config["top_k"]
    ep = runtime.EpMoe(model, batch)
    res = _batch(H, batch)
    got = ep.layer(layer, res)
    want, routed = _oracle_rows(preset, 2, layer, res)
    assert np.array_equal(ep.read("sel_idx", np.int32).reshape(batch, k + 1)[:, :k], routed)
    assert np.array_equal(got, want)
    counts = ep.read("counts", np.int32)
    n_down = counts[2] + counts[4]                       # experts with few rows + experts with many
    assert counts[0] == batch * k and counts[1] + counts[3] == 2 * n_down
    assert 1 <= n_down <= min(model.config["experts"], batch * k) + 1   # + the shared expert
    # a second layer through the same object, chained (res <- x), equals two oracle layers
    if model.config["text_layers"] > layer + 1:
        ep.write("res", res)
        ep.stack(layer, 2)
        dev.sync()
        want2, _ = _oracle_rows(preset, 2, layer + 1, want)
        assert np.array_equal(ep.read("x", np.float32).reshape(batch, H), want2)
    ep.close(); model.close(); dev.close()


@pytest.mark.parametrize("batch", [3, 8, 9, 100])
def test_counts_by_rows_of_an_expert(batch):
    """The "counts" buffer: items, problems of experts with at most eight rows, of experts with more (cut at 64), and of both."""
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, "synth:tiny:seed=2")
    k = model.config["top_k"]
    ep = runtime.EpMoe(model, batch)
    ep.layer(0, _batch(model.config["hidden"], batch))
    routed = ep.read("sel_idx", np.int32).reshape(batch, k + 1)[:, :k]
    rows = np.append(np.bincount(routed.ravel(), minlength=model.config["experts"]), batch)     # the shared expert has them all
    few, every = int(((rows > 0) & (rows <= 8)).sum()), sum(-(-int(c) // 64) for c in rows)
    assert ep.read("counts", np.int32).tolist()[:7] == [batch * k, 2 * few, few, 2 * (every - few), every - few, 2 * every, every]
    ep.close(); model.close(); dev.close()


# mean rows of an expert 8 and just above, 20 and just above, and 24: problems of 16, 32 and 64 rows
@pytest.mark.parametrize("batch", [128, 129, 320, 321, 384])
def test_problems_of_every_cut(batch):
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, "synth:tiny:seed=2")
    ep = runtime.EpMoe(model, batch)
    res = _batch(model.config["hidden"], batch, seed=batch)
    got = ep.layer(1, res)
    want, _ = _oracle_rows("tiny", 2, 1, res)
    assert np.array_equal(got, want)
    ep.close(); model.close(); dev.close()


# the cut at, above and below the rows of an expert, and counts by 64 rows beside lists cut by fewer
@pytest.mark.parametrize("n,k,E,cut,shared", [(1, 3, 32, 1, 1), (9, 3, 40, 5, 9), (100, 11, 32, 16, 0), (130, 4, 1024, 32, 130), (744, 11, 64, 64, 744), (2048, 4, 96, 64, 7)])
@pytest.mark.parametrize("name", ["EpGroupLocal", "EpGroupLocalCut"])
def test_grouping_of_one_rank(name, n, k, E, cut, shared):
    """Items by expert, their places, and the problem lists; EpGroupLocal counts the problems by its own cut, EpGroupLocalCut by 64 rows."""
    from ainfer_b200 import cuda_abi
    dev = cuda_abi.Device(0)
    rng = np.random.default_rng(n)
    p = 1.0 / (1 + np.arange(E)); p /= p.sum()
    sel = np.stack([np.append(rng.choice(E, k, replace=False, p=p), E) for _ in range(n)]).astype(np.int32)
    tab = (np.arange((E + 1) * 6, dtype=np.uint64) + 1) * 256           # weights' addresses: not followed here
    items, rows = n * k, np.bincount(sel[:, :k].ravel(), minlength=E)
    start, I, row0 = np.cumsum(rows) - rows, 128, n * k
    want = [(e, int(start[e]) + j, min(cut, int(rows[e]) - j)) for e in range(E) for j in range(0, int(rows[e]), cut)]
    want += [(E, row0 + j, min(cut, shared - j)) for j in range(0, shared, cut)]
    by = cut if name == "EpGroupLocal" else 64
    every, few = sum(-(-int(c) // by) for c in (*rows, shared)), int(((rows > 0) & (rows <= 8)).sum()) + (0 < shared <= 8)
    dsorted, dplace, gu, gd, counts, lists = (dev.zeros(b) for b in (items * 4, items * 4, 64 * len(want), 32 * len(want), 32, 16))
    dev.kernel(name)(1, dev.upload(sel), dev.upload(tab), dsorted, dplace, gu, gd, counts, n, k, E, I, row0, shared, cut,
                     *([lists] if name == "EpGroupLocalCut" else []))
    dev.sync()
    got, place = dev.download(dsorted, items, np.int32), dev.download(dplace, items, np.int32)
    flat = sel[:, :k].ravel()
    assert np.array_equal(np.sort(got), np.arange(items)) and np.array_equal(got[place], np.arange(items)) and (np.diff(flat[got]) >= 0).all()
    assert dev.download(counts, 8, np.int32).tolist() == [items, 2 * few, few, 2 * (every - few), every - few, 2 * every, every, 0]
    if name == "EpGroupLocalCut":
        assert dev.download(lists, 2, np.int32).tolist() == [2 * len(want), len(want)]
    kind = np.dtype([("P", "<u8"), ("S", "<u8"), ("row0", "<i4"), ("M", "<i4"), ("col", "<i4"), ("pad", "<i4")])
    t = tab.reshape(E + 1, 6)
    down, gate_up = dev.download(gd, 32 * len(want), np.uint8).view(kind), dev.download(gu, 64 * len(want), np.uint8).view(kind)
    assert [tuple(x)[:5] for x in down.tolist()] == [(int(t[e, 4]), int(t[e, 5]), r, m, 0) for e, r, m in want]
    assert [tuple(x)[:5] for x in gate_up.tolist()] == [(int(t[e, 2 * u]), int(t[e, 2 * u + 1]), r, m, u * I) for e, r, m in want for u in (0, 1)]
    dev.close()


@pytest.mark.parametrize("world,n,cut", [(2, 20, 16), (4, 3, 64), (2, 40, 64), (1, 9, 5)])
def test_kernels_of_several_ranks_one_after_the_other(world, n, cut):
    """Plan, pack, group, gather, both grouped products, scatter and combine of every rank, one rank after the other on one
    GPU with copies in the exchanges' place, against the oracle's products and sums: every row bit for bit."""
    from ainfer_b200 import cuda_abi
    L = O.lib()
    dev = cuda_abi.Device(0)
    rng = np.random.default_rng(world * 100 + n)
    E, k, H, I = 16, 3, 256, 128
    epr, cap = E // world, n * k
    item, rows = H + ((H // 128 * 4 + 15) & ~15), world * n * k
    slot_d, slot_r = (16 + cap * 16 + cap * item + 15) & ~15, cap * H * 4
    W = [[O.quantize_int4((rng.standard_normal(sh) * 0.05).astype(np.float32)) for sh in ((I, H), (I, H), (H, I))] for _ in range(E + 1)]
    tab = np.zeros((E + 1, 6), np.uint64)
    for e in range(E + 1):
        tab[e] = [dev.upload(a) for w in W[e] for a in w]
    d_tab = dev.upload(tab.view(np.uint8))

    def expert(e, q, s):
        g, u = O.gemv_a8(*W[e][0], q, s), O.gemv_a8(*W[e][1], q, s)
        act = np.array([(a / (np.float32(1.0) + np.float32(L.orc_expf(float(-a))))) * b for a, b in zip(g, u)], np.float32)
        return O.gemv_a8(*W[e][2], *O.aquant(act))
    p = np.exp(-0.3 * np.arange(E)); p /= p.sum()          # a few experts get most rows
    ranks = []
    for r in range(world):
        x, res = rng.standard_normal((n, H)).astype(np.float32), rng.standard_normal((n, H)).astype(np.float32)
        q = [O.aquant(v) for v in x]
        sel = np.array([np.append(rng.choice(E, k, replace=False, p=p), E) for _ in range(n)], np.int32)
        sw = rng.random((n, k + 1)).astype(np.float32)
        want = np.zeros((n, H), np.float32)
        for t in range(n):
            acc = np.zeros(H, np.float32)
            for j in range(k + 1):
                acc = acc + sw[t, j] * expert(int(sel[t, j]), *q[t])
            want[t] = res[t] + acc
        d = dict(want=want, sel=dev.upload(sel), sw=dev.upload(sw), res=dev.upload(res), dest=dev.zeros(cap * 4), send=dev.zeros(world * slot_d),
                 recv=dev.zeros(world * slot_d), ret=dev.zeros(world * slot_r), back=dev.zeros(world * slot_r), sorted=dev.zeros(rows * 4),
                 counts=dev.zeros(32), gu=dev.zeros(64 * (2 * rows + 64)), gd=dev.zeros(64 * (rows + 64)), xq=dev.zeros((rows + n) * H),
                 xs=dev.zeros((rows + n) * (H // 128) * 4), h=dev.zeros((rows + n) * 2 * I * 4), aq=dev.zeros((rows + n) * I),
                 as_=dev.zeros((rows + n) * (I // 128) * 4), y=dev.zeros((rows + n) * H * 4), x=dev.zeros(n * H * 4))
        d["q8"], d["sq"] = d["xq"] + rows * H, d["xs"] + rows * (H // 128) * 4
        dev.write(d["q8"], np.stack([a for a, _ in q])); dev.write(d["sq"], np.stack([b for _, b in q]))
        dev.kernel("EpPlan")(1, d["sel"], d["send"], d["dest"], n, k, epr, world, cap, slot_d)
        dev.kernel("EpPack")(cap, d["q8"], d["sq"], d["dest"], d["send"], k, H, cap, slot_d)
        ranks.append(d)

    def exchange(src, dst, slot):
        for a in range(world):
            for b in range(world):
                dev.copy_d2d(ranks[b][dst] + a * slot, ranks[a][src] + b * slot, slot)
    exchange("send", "recv", slot_d)
    for r, d in enumerate(ranks):
        dev.kernel("EpGroup")(1, d["recv"], d_tab, d["sorted"], d["gu"], d["gd"], d["counts"], world, r, epr, cap, I, slot_d, rows, n, E, cut)
        dev.kernel("EpGather")(rows, d["recv"], d["sorted"], d["counts"], d["xq"], d["xs"], H, cap, slot_d)
        grouped = dev.kernel("Int4GemmA8TcGrouped")
        grouped(37, d["gu"], d["counts"] + 20, d["xq"], d["xs"], d["h"], I, H, cut, 2 * I)
        dev.kernel("SiluQuantRows")(rows + n, d["h"], d["counts"], d["aq"], d["as_"], I, rows, rows)
        grouped(37, d["gd"], d["counts"] + 24, d["aq"], d["as_"], d["y"], H, I, cut, H)
        dev.kernel("EpScatter")(rows, d["y"], d["sorted"], d["counts"], d["ret"], H, slot_r)
    exchange("ret", "back", slot_r)
    received = 0
    for d in ranks:
        dev.kernel("EpCombine")(n * -(-H // 256), d["res"], d["back"], d["dest"], d["sw"], d["y"] + rows * H * 4, d["x"], d["res"], k, H, slot_r)
        dev.sync()
        assert np.array_equal(dev.download(d["x"], (n, H), np.float32), d["want"])
        assert np.array_equal(dev.download(d["res"], (n, H), np.float32), d["want"])
        received += int(dev.download(d["counts"], 8, np.int32)[0])
    assert received == world * cap
    dev.close()


def test_usage_errors():
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, "synth:tiny:seed=0")
    for kw in (dict(batch=3, world=2), dict(batch=4096), dict(batch=4, world=2, rank=0)):   # ragged split, too many (row, expert) items, no id
        with pytest.raises(Exception) as e:
            runtime.EpMoe(model, **kw)
        assert "usage" in str(e.value)
    model.close(); dev.close()


def test_the_planner_of_prompt_passes_is_not_asked_for_by_a_flag():
    """The documented limit of batch x top-k holds whatever other bits a caller sets."""
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, "synth:tiny:seed=0")
    for bit in range(2, 12):
        with pytest.raises(Exception) as e:
            runtime.EpMoe(model, 1025, flags=1 << bit)
        assert "usage" in str(e.value)
    runtime.EpMoe(model, 1024, flags=4).close()
    model.close(); dev.close()


def _rank_main(rank, world, conn, q, preset, batch, layer):
    os.environ["NCCL_NVLS_ENABLE"] = "0"
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(rank)
    if rank == 0:
        nid = runtime.ep_unique_id()
        for c in conn:
            c.send_bytes(nid)
    else:
        nid = conn[0].recv_bytes()
    model = runtime.Model(dev, f"synth:{preset}:seed=2")       # replicated weights: same seed on every rank
    H = model.config["hidden"]
    ep = runtime.EpMoe(model, batch, rank=rank, world=world, nccl_id=nid)
    n = batch // world
    res = _batch(H, batch)[rank * n:(rank + 1) * n]
    out = ep.layer(layer, res)
    seg = ep.stack(layer, 1, segments=True)
    q.put((rank, out, ep.read("counts", np.int32), seg))
    ep.close(); model.close(); dev.close()


@pytest.mark.parametrize("preset,batch,layer", [("mini", 16, 1), ("small", 64, 1)])
def test_two_nccl_ranks_equal_oracle(preset, batch, layer):
    from ainfer_b200 import cuda_abi
    if cuda_abi.device_count() < 2:
        pytest.skip("needs two GPUs")
    import multiprocessing as mp
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    a, b = ctx.Pipe()
    procs = [ctx.Process(target=_rank_main, args=(0, 2, [a], q, preset, batch, layer)),
             ctx.Process(target=_rank_main, args=(1, 2, [b], q, preset, batch, layer))]
    for p in procs:
        p.start()
    got = {}
    for _ in procs:
        r, out, counts, seg = q.get(timeout=600)
        got[r] = (out, counts, seg)
    for p in procs:
        p.join(120)
        assert p.exitcode == 0
    import json
    H = json.loads(O.preset_json(preset))["hidden"]
    k = json.loads(O.preset_json(preset))["top_k"]
    want, _ = _oracle_rows(preset, 2, layer, _batch(H, batch))
    n = batch // 2
    assert np.array_equal(got[0][0], want[:n]) and np.array_equal(got[1][0], want[n:])
    assert got[0][1][0] + got[1][1][0] == batch * k          # every (token, slot) item computed exactly once
    print(json.dumps({"ep_two_ranks": {"preset": preset, "batch": batch, "items": [int(got[0][1][0]), int(got[1][1][0])],
                                       "segments_ms_rank0": [round(x, 4) for x in got[0][2]]}}))
