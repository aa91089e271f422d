"""Logits of decode steps, bit for bit from one version to the next. An output in 16 bits carries a last bit of a layer's sums through
all layers that follow, and a mixture then chooses another expert: a batch's logits move by a percent when the cut of its keys or the
order of a merge does. So the order is held here, by checksums of what the first version with this cut gave on a B200."""
import tempfile
import zlib

import numpy as np
import pytest

import robopel_plain as R
import sinepel_plain as S

pytestmark = pytest.mark.gpu

L = S.make_layer
MODELS = {
    "sinepel": S.make_config(width=256, vocab=320, streams=4, max_positions=1024,
                             layers=[L(heads=16, kv_heads=4, dim=64, conv=4, chunk=700, ff=512), L(heads=8, kv_heads=2, dim=128, conv=3, chunk=260, ff=256)]),
    "robopel": R.make_config(width=256, vocab=320, layers=[
        R.attention(heads=16, kv_heads=4, dim=64, vdim=64, size=400, pool=16, turn=R.rot(64, 1e4), softcap=30.0, mlp=R.dense(512)),
        R.mingru(256, R.moe(8, 2, 3, 128)),
        R.attention(heads=8, kv_heads=4, dim=64, vdim=64, size=300, pool=16, turn=R.rot(64, 1e4), softcap=30.0, kv_from=0)]),
}
LAST = (4, 130, 470)       # one tile of keys, a few, eight: one and several shares of a head
WANT = {
    ("sinepel", 1): [831997823, 1813388974, 2380410665], ("sinepel", 5): [835060282, 1637585199, 708969669],
    ("sinepel", 16): [1517585307, 4209787457, 3551985280], ("sinepel", 64): [1161367069, 304899933, 2391206509],
    ("robopel", 1): [4052954358, 4251945721, 1144347737], ("robopel", 5): [735788599, 2280388135, 1378504494],
    ("robopel", 16): [1382367426, 818599329, 1609085430], ("robopel", 64): [3843409105, 2792703231, 168510517],
}


def digests(arch, seqs):
    from ainfer_b200 import cuda_abi, runtime
    c, p = MODELS[arch], S if arch == "sinepel" else R
    dev = cuda_abi.Device(0)
    with tempfile.TemporaryDirectory() as folder:
        p.write_model(folder, c, p.make_weights(c, 11))
        model = runtime.Model(dev, folder)
    ids = np.random.default_rng(seqs).integers(0, c["vocab"], (LAST[-1] + 1, seqs)).astype(np.int32)
    s = runtime.BatchDecode(model, seqs, 480) if seqs > 1 else runtime.Session(model, 480)
    got = []
    for i in range(LAST[-1] + 1):
        if seqs > 1:
            s.set_inputs(ids[i], np.full(seqs, i, np.int32))
            s.step()
        else:
            s.step(int(ids[i, 0]), i)
        if i in LAST:
            dev.sync()
            got.append(zlib.crc32(s.read("logits", np.float32).tobytes()))
    s.close()
    model.close()
    dev.close()
    return got


@pytest.mark.parametrize("arch,seqs", [(a, n) for a in ("sinepel", "robopel") for n in (1, 5, 16, 64)])
def test_logits_keep_their_bits(arch, seqs):
    assert digests(arch, seqs) == WANT[arch, seqs]
