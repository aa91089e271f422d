"""The persistent step's hand-overs and attention at their edges: against the recorded list's kernels, bit for bit. Its quantiser
against the oracle's. A wait of it that runs out."""
import json

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


def _run(model, flags, ctx, fill, prompt, start, steps):
    from ainfer_b200 import runtime
    s = runtime.Session(model, ctx, flags)
    s.reset()
    rng = np.random.default_rng(3)
    for name in ("Kc", "Vc", "Ks", "Vs", "S", "conv"):
        n = s.buffer(name)[1]
        if fill and n:
            raw = (rng.integers(-127, 128, n, np.int64).astype(np.int8) if name in ("Kc", "Vc") else
                   (0.008 + 0.008 * rng.random(n // 2)).astype(np.float16) if name in ("Ks", "Vs") else
                   (0.1 * rng.standard_normal(n // 4)).astype(np.float32))
            s.write(name, raw)
    tokens = s.generate(np.asarray(prompt, np.int32), steps, start_pos=start)
    out = {"tokens": tokens, "logits": s.logits()}
    for name, t in (("x", np.float32), ("S", np.float32), ("conv", np.float32), ("Kc", np.int8), ("Vc", np.int8), ("Ks", np.uint16), ("Vs", np.uint16)):
        out[name] = s.read(name, t)
    s.close()
    return out


# tiny: more blocks than units of rows; chunk edges of the attention, and more chunks than the merge takes at a time
@pytest.mark.parametrize("preset,prompt,start,steps", [("tiny", 3, 0, 70), ("mini", 61, 0, 8), ("mini", 1, 64, 1), ("mini", 2, 126, 4),
                                                       ("tiny", 1, 4095, 3), ("mini", 1, 8190, 4), ("small", 2, 255, 3)])
def test_persistent_step_equals_list(preset, prompt, start, steps):
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, f"synth:{preset}:seed=5")
    ids = (np.arange(prompt) * 131 + 7) % model.config["vocab"]
    ctx = start + prompt + steps + 1
    got, want = (_run(model, f, ctx, start > 0, ids, start, steps) for f in (runtime.Session.PERSISTENT, runtime.Session.MULTI_KERNEL))
    for name in want:
        assert np.array_equal(got[name], want[name]), name
    model.close()
    dev.close()


# An odd number of layers: a launch begins in the set of words that the last one ended in. A second run of 512 experts, the most and
# the fewest chosen, no shared expert; rows of 32 groups; a query head for each key head; one layer alone of either type.
@pytest.mark.parametrize("over", [
    dict(hidden=4096, experts=1024, top_k=11, shared_experts=0, q_heads=4, kv_heads=4),
    dict(hidden=256, experts=32, top_k=11, q_heads=2, kv_heads=2, lin_k_heads=1, lin_v_heads=1),
    dict(text_layers=5, layer_types="ALLAA", experts=544, top_k=1, hidden=512), dict(text_layers=1, layer_types="A", hidden=2048, q_heads=16, kv_heads=8),
    dict(text_layers=1, layer_types="L", lin_k_heads=32, lin_v_heads=32, expert_intermediate=512)])
def test_persistent_step_of_other_shapes_equals_list(tmp_path, over):
    from ainfer_b200 import cuda_abi, runtime
    f = tmp_path / "model.json"
    f.write_text(json.dumps({**json.loads(runtime.preset_config_json("mini")), "text_layers": 3, "layer_types": "LAL", "vocab": 1000,
                             "expert_intermediate": 128, **over}))
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, f"synth:config:{f}:seed=5")
    ids = (np.arange(5) * 131 + 7) % model.config["vocab"]
    for start in (0, 200):
        got, want = (_run(model, fl, start + 20, start > 0, ids, start, 9) for fl in (runtime.Session.PERSISTENT, runtime.Session.MULTI_KERNEL))
        for name in want:
            assert np.array_equal(got[name], want[name]), (start, name)
    model.close()
    dev.close()


def test_quantiser_of_a_group():
    """Quotients on half-integers and next to them, on either side of the margin from which the division decides; maxima from subnormal to
    the largest; groups of zeros, with an infinity, with a NaN."""
    from ainfer_b200 import cuda_abi
    rng = np.random.default_rng(1)
    near = np.array([0, 1e-7, 1e-6, 5e-6, 2e-5, 5e-5, 7e-5, 8e-5, 9e-5, 1.2e-4, 2e-4, 0.3])
    near = np.concatenate([near, -near])
    groups = [np.zeros(128, np.float32)]
    for e in list(range(-148, 129)) + [0] * 400:
        mx = np.float32(np.ldexp(rng.uniform(0.5, 0.999), e))
        s = float(mx / np.float32(127.0))
        x = np.float32((rng.integers(0, 127, 128) + 0.5 + rng.choice(near, 128)) * s) * rng.choice([-1, 1], 128).astype(np.float32)
        x = np.clip(x, -mx, mx)
        x[rng.integers(128)] = mx * rng.choice([-1, 1])
        groups.append(x)
    odd = np.zeros((2, 128), np.float32)
    odd[0, :3] = np.inf, -3.0, 1e38            # an infinite scale: every quotient is zero or no number, both zero
    odd[1, :4] = np.nan, 5.0, -5.0, 2.5        # no part of the maximum, and zero
    x = np.concatenate([np.stack(groups).astype(np.float32), odd])
    want = [O.aquant(v) for v in np.nan_to_num(x[:-2])] + [(np.zeros(128, np.int8), np.full(1, np.inf)), O.aquant(np.nan_to_num(odd[1]))]
    dev = cuda_abi.Device(0)
    n = len(x)
    q, s = dev.zeros(n * 128), dev.zeros(n * 4)
    dev.kernel("StepQuantGroups")(-(-n // 4), dev.upload(x), q, s, n)
    dev.sync()
    assert np.array_equal(dev.download(s, n, np.float32), np.concatenate([w for _, w in want]).astype(np.float32))
    assert np.array_equal(dev.download(q, (n, 128), np.int8), np.stack([w for w, _ in want]))
    dev.close()


def test_a_wait_that_runs_out_is_reported():
    """A count of arrivals that never reaches its target: the step ends by itself and says so, and so does every later one of the
    session; other sessions go on."""
    from ainfer_b200 import cuda_abi, runtime
    dev = cuda_abi.Device(0)
    model = runtime.Model(dev, "synth:tiny:seed=5")
    good, bad = (runtime.Session(model, 32, runtime.Session.PERSISTENT) for _ in range(2))
    first = good.step(3, 0)
    assert bad.step(3, 0) == first
    sync = bad.read("step_sync", np.uint32)
    sync[1] += 1 << 20                        # the count when the launch starts: more than there were
    bad.write("step_sync", sync)
    for pos in (1, 2):
        with pytest.raises(Exception, match="bounded wait of the persistent decode kernel ran out"):
            bad.step(first, pos)
    other = runtime.Session(model, 32, runtime.Session.MULTI_KERNEL)
    assert other.step(3, 0) == first
    assert good.step(first, 1) == other.step(first, 1)
    for s in (good, bad, other):
        s.close()
    model.close()
    dev.close()
