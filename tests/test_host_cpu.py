"""Host-side tests that need no GPU: the C-ABI libraries load and export every
declared symbol, the container writer/validator agree with the oracle's parser
(and with the reference's own validator when its checkout is present), the
reference's negative container cases are rejected, the host sampler reproduces
the reference sampler's outputs, and the CLI keeps the reference's exit codes."""
import ctypes as C
import importlib.util
import json
import os
import re
import struct
import subprocess

import numpy as np
import pytest

import oracle_lib as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
G = os.path.join(os.path.dirname(__file__), "golden")
REF = os.environ.get("REFERENCE") or os.path.join(os.path.dirname(ROOT), "reference")


@pytest.fixture(scope="session", autouse=True)
def built():
    from ainfer_b200 import _build
    _build.build_all()


@pytest.fixture(scope="module")
def tiny_file(tmp_path_factory):
    from ainfer_b200 import runtime
    p = str(tmp_path_factory.mktemp("m") / "tiny.binfer")
    runtime.synth_write(p, "tiny", seed=0)
    return p


def declared_symbols(header):
    txt = open(os.path.join(ROOT, "include", header)).read()
    txt = re.sub(r"/\*.*?\*/", "", txt, flags=re.S)
    return sorted(set(re.findall(r"\b(ainfer_[a-z0-9_]+)\s*\(", txt)))


def test_libraries_export_every_declared_symbol():
    from ainfer_b200 import cuda_abi, runtime
    Lc, Lr = cuda_abi.load(), runtime.load()
    cu = declared_symbols("ainfer_cuda.h")
    rt = declared_symbols("ainfer_runtime.h")
    assert len(cu) >= 35 and len(rt) >= 18
    for s in cu:
        assert hasattr(Lc, s), s
        assert s in cuda_abi.SIGNATURES, f"{s} has no ctypes signature"
    for s in rt:
        assert hasattr(Lr, s), s
        assert s in runtime.SIGNATURES, f"{s} has no ctypes signature"
    names = [Lc.ainfer_kernel_name(i).decode() for i in range(Lc.ainfer_kernel_count())]
    for k in ["Int4GemvA8", "RmsNormQuant", "DeltaNetStep", "GatedNormQuant", "AttnPrep", "AttnSplit",
              "AttnCombine", "RouterTopK", "ExpertGateUp", "ExpertDownCombine", "EmbedRow",
              "ArgmaxStage1", "ArgmaxStage2", "ControlAdvance", "SynthInt4", "SynthBf16"]:
        assert k in names


def test_no_gpu_means_loud_failure_not_fallback():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    from ainfer_b200 import cuda_abi
    with pytest.raises(cuda_abi.AinferError) as e:
        cuda_abi.Device(0)
    assert e.value.status == 4 and "no CPU fallback" in str(e.value)


def test_synth_container_validates_and_matches_oracle(tiny_file):
    from ainfer_b200 import runtime
    rc, msg = runtime.validate(tiny_file, 2)
    assert rc == 0, msg
    m = O.Model(path=tiny_file, check_crc=True)
    cfg = json.loads(m.arch_json)
    assert cfg == json.loads(runtime.preset_config_json("tiny"))
    # every tensor kind regenerated by the oracle's generator + quantiser: bit-exact
    for name, std in [("lm_head.weight", 0.02),
                      ("model.language_model.layers.0.linear_attn.in_proj_qkv.weight", 0.02),
                      ("model.language_model.layers.1.mlp.experts.7.down_proj.weight", 0.02),
                      ("mtp.fc.weight", 0.02)]:
        t = m.tensor(name)
        n = int(np.prod(t["shape"]))
        P, S = O.quantize_int4(O.synth_normal(name, 0, n, std))
        assert t["storage"] == 3
        assert np.array_equal(t["data"], P.reshape(-1)), name
        assert np.array_equal(t["scales"], S.reshape(-1)), name
    for name, std in [("model.language_model.embed_tokens.weight", 0.02),
                      ("model.language_model.layers.0.linear_attn.conv1d.weight", 0.5),
                      ("model.language_model.layers.0.linear_attn.A_log", 0.05),
                      ("model.language_model.layers.1.mlp.gate.weight", 0.02)]:
        t = m.tensor(name)
        n = int(np.prod(t["shape"]))
        assert t["storage"] == 0
        assert np.array_equal(t["data"].view(np.uint16), O.bf16_bits(O.synth_normal(name, 0, n, std))), name
    assert np.all(m.tensor("model.language_model.layers.0.input_layernorm.weight")["data"] == 0)
    ones = m.tensor("model.language_model.layers.0.linear_attn.norm.weight")["data"].view(np.uint16)
    assert np.all(ones == 0x3F80)
    m.close()


@pytest.mark.skipif(not os.path.isfile(os.path.join(REF, "tools", "binfer.py")), reason="reference checkout not present")
def test_reference_validator_accepts_our_container(tiny_file, capsys):
    spec = importlib.util.spec_from_file_location("ref_binfer", os.path.join(REF, "tools", "binfer.py"))
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    assert mod.cmd_validate(tiny_file) == 0
    assert "VALID" in capsys.readouterr().out


def _mutated(src, dst, fn):
    data = bytearray(open(src, "rb").read())
    data = fn(data)
    open(dst, "wb").write(data)
    return dst


def test_container_negative_cases(tiny_file, tmp_path):
    """The reference's negative set (tools/binfer.py:502-622): bad magic, bad version,
    truncation, payload CRC flip, unknown layout id; plus span overflow (decode_l0.cpp:176-189)."""
    from ainfer_b200 import runtime
    size = os.path.getsize(tiny_file)
    raw = open(tiny_file, "rb").read()
    dir_off = None
    n_tensors = struct.unpack_from("<Q", raw, 16)[0]
    table_off = struct.unpack_from("<Q", raw, 24)[0]
    for i in range(5):
        sid, off, nb, crc, _, _ = struct.unpack_from("<I2Q3I", raw, table_off + 32 * i)
        if sid == 5:
            dir_off = off
    first_payload = struct.unpack_from("<Q", raw, dir_off + 160)[0]

    def case(name, fn, level, expect):
        p = _mutated(tiny_file, str(tmp_path / f"{name}.binfer"), fn)
        rc, msg = runtime.validate(p, level)
        assert rc == 2 and expect in msg, (name, rc, msg)
        with pytest.raises(ValueError):
            O.Model(path=p, check_crc=True)

    def bad_magic(d): d[0:4] = b"XXXX"; return d
    def bad_version(d): struct.pack_into("<I", d, 8, 2); return d
    def truncated(d): return d[: size // 2]
    def crc_flip(d): d[first_payload + 5] ^= 0xFF; return d
    def bad_layout(d):
        struct.pack_into("<H", d, dir_off + 138, 99)
        struct.pack_into("<I", d, table_off + 32 * 4 + 20, O.lib().orc_crc32(
            np.frombuffer(bytes(d[dir_off:dir_off + n_tensors * 192]), np.uint8), n_tensors * 192))
        return d
    def span_overflow(d):
        struct.pack_into("<Q", d, dir_off + 168, size)   # d_bytes beyond the file
        return d

    case("magic", bad_magic, 0, "bad magic (not a .binfer file)")
    case("version", bad_version, 0, "bad version")
    case("trunc", truncated, 0, "total mismatch")
    case("crc", crc_flip, 2, "payload CRC")
    case("layout", bad_layout, 0, "unsupported layout_id")
    case("span", span_overflow, 0, "payload span out of range")
    rc, _ = runtime.validate(tiny_file, 2)
    assert rc == 0
    rc, msg = runtime.validate(str(tmp_path / "nope.binfer"), 0)
    assert rc == 2


def test_host_sampler_matches_reference_golden():
    from ainfer_b200 import runtime
    g = json.load(open(os.path.join(G, "sampler_golden.json")))
    logits = np.array(g["logits"], np.float32)
    for c in g["cases"]:
        lg = logits.copy()
        if c["rep_penalty"] > 1.0:
            lg = runtime.apply_rep_penalty(lg, c["seen"], c["rep_penalty"])
        assert np.array_equal(lg, np.array(c["penalised_logits"], np.float32))
        state = c["rng_init"]
        toks = []
        for _ in range(len(c["tokens"])):
            t, state, probs = runtime.sample_token(lg, c["temp"], c["top_k"], c["top_p"], c["rep_penalty"],
                                                   c["seed"], rng=state, want_probs=True)
            toks.append(t)
        assert toks == c["tokens"], c
        assert state == c["rng_final"]
        assert np.array_equal(probs, np.array(c["probs"], np.float32))
    # greedy: planted tie -> the first maximum wins
    assert g["cases"][0]["tokens"][0] == 11


@pytest.mark.skipif(not os.path.isfile(os.path.join(REF, "tools", "sample", "validate_t71.cpp")), reason="reference checkout not present")
def test_host_sampler_matches_reference_live():
    """Fresh random cases through the reference's own sampler (oracle/_ref) and ours."""
    from ainfer_b200 import runtime
    subprocess.run(["make", "-C", os.path.join(ROOT, "oracle"), "ref", f"REFERENCE={REF}"], check=True,
                   stdout=subprocess.DEVNULL)
    R = C.CDLL(os.path.join(ROOT, "oracle", "_ref", "libref_sampler.so"))
    f32p = np.ctypeslib.ndpointer(np.float32, flags="C_CONTIGUOUS")
    R.ref_sample_token.restype = C.c_int
    R.ref_sample_token.argtypes = [f32p, C.c_int, C.c_float, C.c_int, C.c_float, C.c_float, C.c_uint64,
                                   C.POINTER(C.c_uint64), C.c_void_p]
    rng = np.random.default_rng(9)
    for trial in range(40):
        V = int(rng.integers(2, 400))
        lg = (rng.standard_normal(V) * rng.uniform(0.5, 4)).astype(np.float32)
        temp = float(rng.choice([0.0, 0.3, 1.0, 1.7]))
        top_k = int(rng.choice([0, 1, 3, V // 2, V + 5]))
        top_p = float(rng.choice([1.0, 0.95, 0.5, 0.01]))
        seed = int(rng.integers(1, 2**62))
        st_ref = C.c_uint64(seed)
        st = seed
        for _ in range(5):
            want = R.ref_sample_token(lg, V, temp, top_k, top_p, 1.0, seed, C.byref(st_ref), None)
            got, st, _ = runtime.sample_token(lg, temp, top_k, top_p, 1.0, seed, rng=st)
            assert got == want and st == st_ref.value, (trial, V, temp, top_k, top_p)


def test_cli_exit_codes(tiny_file, tmp_path):
    from ainfer_b200 import runtime
    exe = runtime.DECODE_EXE
    assert os.path.exists(exe)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 2 and "usage" in r.stderr
    import torch
    if not torch.cuda.is_available():
        r = subprocess.run([exe, tiny_file, "4", "4"], capture_output=True, text=True)
        assert r.returncode == 2 and "no CPU fallback" in r.stderr


def test_presets_describe_the_baseline_shapes():
    from ainfer_b200 import runtime
    mini = json.loads(runtime.preset_config_json("mini"))
    assert (mini["hidden"], mini["layer_types"], mini["experts"], mini["top_k"], mini["expert_intermediate"],
            mini["vocab"], mini["q_heads"], mini["kv_heads"], mini["lin_k_heads"], mini["lin_v_heads"]) == \
        (1024, "LA", 64, 4, 256, 32000, 8, 2, 8, 16)
    full = json.loads(runtime.preset_config_json("full"))
    assert full["text_layers"] == 48 and full["layer_types"] == "LLLA" * 12
    assert (full["hidden"], full["experts"], full["top_k"], full["expert_intermediate"], full["vocab"],
            full["q_heads"], full["kv_heads"], full["lin_k_heads"], full["lin_v_heads"], full["mtp_layers"]) == \
        (2048, 512, 10, 512, 151936, 16, 2, 16, 32, 1)
    assert runtime.preset_config_json("nope") is None


def _dir_entries(raw):
    """(offset of the 192-byte record, name) of every directory entry of a .binfer image."""
    table_off = struct.unpack_from("<Q", raw, 24)[0]
    scount = struct.unpack_from("<I", raw, 32)[0]
    for i in range(scount):
        sid = struct.unpack_from("<I", raw, table_off + 32 * i)[0]
        off, nb = struct.unpack_from("<QQ", raw, table_off + 32 * i + 4)
        if sid == 5:
            return [(off + 192 * j, raw[off + 192 * j:off + 192 * j + 64].split(b"\0")[0].decode())
                    for j in range(nb // 192)]
    raise AssertionError("no directory section")


def test_directory_that_disagrees_with_the_architecture_is_rejected(tiny_file, tmp_path):
    """A container whose directory is self-consistent but smaller than its architecture section
    says (which would make the expert, router and embedding kernels read past the weight arenas)
    is refused on the host, before any upload; so is a payload shorter than its shape."""
    from ainfer_b200 import runtime
    good = bytearray(open(tiny_file, "rb").read())
    ents = dict((n, o) for o, n in _dir_entries(good))
    cases = []
    # an expert matrix with half its rows, packed and scale sizes patched to match the new shape
    raw = bytearray(good)
    o = ents["model.language_model.layers.0.mlp.experts.3.gate_proj.weight"]
    rows, cols = struct.unpack_from("<QQ", raw, o + 72)
    struct.pack_into("<Q", raw, o + 72, rows // 2)
    ng = (rows // 2) * cols // 128
    struct.pack_into("<Q", raw, o + 152, ng * 2)
    struct.pack_into("<Q", raw, o + 168, ng * 64)
    cases.append((raw, "unexpected shape of model.language_model.layers.0.mlp.experts.3.gate_proj.weight"))
    # the router stored as INT4 instead of bf16 (the router kernel reads bf16 rows)
    raw = bytearray(good)
    o = ents["model.language_model.layers.1.mlp.gate.weight"]
    rows, cols = struct.unpack_from("<QQ", raw, o + 72)
    ng = rows * cols // 128
    raw[o + 137] = 3
    struct.pack_into("<I", raw, o + 140, 128)
    d_off = struct.unpack_from("<Q", raw, o + 160)[0]
    struct.pack_into("<QQ", raw, o + 144, d_off, ng * 2)
    struct.pack_into("<Q", raw, o + 168, ng * 64)
    cases.append((raw, "unexpected storage of model.language_model.layers.1.mlp.gate.weight"))
    # a bf16 payload shorter than its shape
    raw = bytearray(good)
    o = ents["model.language_model.embed_tokens.weight"]
    nbytes = struct.unpack_from("<Q", raw, o + 168)[0]
    struct.pack_into("<Q", raw, o + 168, nbytes // 2)
    cases.append((raw, "payload size does not match shape: model.language_model.embed_tokens.weight"))
    for i, (raw, want) in enumerate(cases):
        p = tmp_path / f"crafted{i}.binfer"
        p.write_bytes(bytes(raw))
        rc, msg = runtime.validate(str(p), 0)      # level 0: the checks the loader itself runs
        assert rc == 2 and want in msg, (rc, msg)
    assert runtime.validate(tiny_file, 0)[0] == 0


def test_oracle_preset_table_equals_runtime_presets():
    """The CPU arm of the benchmark takes its model shapes from oracle/presets.json (it must not
    load the product libraries); the table has to stay equal to the runtime's presets."""
    from ainfer_b200 import runtime
    for name in ("tiny", "mini", "mini-mtp", "small", "full"):
        assert json.loads(O.preset_json(name)) == json.loads(runtime.preset_config_json(name)), name


# what a model holds: written once, before any launch that reads it
CONSTANT_FIELDS = {"W", "CW", "Wr", "Wsg", "Bias", "Experts", "P", "S", "LB"}


EARLY_SOURCES = sorted(f for f in os.listdir(os.path.join(ROOT, "ainfer_b200", "csrc", "kernels"))
                       if f.endswith(".cu") and re.search(r"^AINFER_EARLY_LAUNCH\(", open(os.path.join(ROOT, "ainfer_b200", "csrc", "kernels", f)).read(), re.M))


@pytest.mark.parametrize("source", EARLY_SOURCES)
def test_early_kernels_read_results_coherently(source):
    """A kernel marked for early launch may be resident while the kernels before it write: what they write must not be
    read through the read-only path (__ldg), which a dependency wait does not order."""
    text = open(os.path.join(ROOT, "ainfer_b200", "csrc", "kernels", source)).read()
    marked = re.findall(r"^AINFER_EARLY_LAUNCH\((\w+)\)", text, re.M)
    assert marked
    for name in marked:
        head = re.search(r"__global__[^;{]*\b%s\(" % name, text)
        if not head:      # made by a macro around a shared body
            continue
        start = text.index("{", head.start())
        depth, end = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        read = set(re.findall(r"__ldg\([^;]*?\ba\.(\w+)", text[start:end]))
        assert read <= CONSTANT_FIELDS, (name, read - CONSTANT_FIELDS)
