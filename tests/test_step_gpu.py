"""The persistent step's hand-overs and attention at their edges: against the recorded list's kernels, bit for bit."""
import numpy as np
import pytest

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
