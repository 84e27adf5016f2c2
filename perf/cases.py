"""The work that a program has this library do, as cases of stated sizes: speech (prompt, first frame, utterances, a
batch, the reference's call sequence), the codec decoder, and the decoder language models (prompts, greedy
continuation, a sampling loop, checking drafted tokens), each through the entry points of the package's bindings.

    listed()            the cases
    draw(rng)           another case of the same ranges
    prepare(case, seed) what a program has in hand before the call
    run(state)          one pass
    work(case)          the bytes and operations that a pass cannot do without
    tolerance(case)     how far two correct implementations may be apart
    exact(case, seed)   the same results in 64 bits, by torch alone

Models are loaded once in a process and kept, as a serving program keeps them; inputs are made from the seed."""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NAME = "voxtral_tts_c_b200"


def package():
    if NAME not in sys.modules:
        folder = os.path.join(ROOT, "voxtral-tts.c_b200")
        spec = importlib.util.spec_from_file_location(NAME, os.path.join(folder, "__init__.py"), submodule_search_locations=[folder])
        sys.modules[NAME] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[NAME])
    return sys.modules[NAME]


# ---------------------------------------------------------------------------------------------- the cases

KV_ROWS = 2048          # cache rows of the speech engine
LM_TOKENS = 4608        # longest sequence of a language-model slot


def _latent_mixer(heads, q_rank, window):
    return {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": q_rank, "scale": 192 ** -0.5,
            "mask": {"size": window}, "rot": {"dims": 64, "base": 100000.0}}


def _kegizen(width, ff, layers, dh, dkv, ah, akv, vocab, window, loop=None):
    mlp = {"kind": "dense", "ff": ff}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": dh, "kv_heads": dkv, "dim": 128, "vdim": 128, "conv": 4}}
    att = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": ah, "kv_heads": akv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
        "mask": {"size": window, "keep_first": 4},
        "rot": {"dims": 64, "base": 100000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    c = {"architecture": "Kegizen", "layers": [delta, att] * (layers // 2), "norm": {"eps": 1e-5}, "vocab": vocab, "width": width}
    if loop:
        c["loop"] = dict(zip(("start", "stop", "times"), loop))
    return c


def _bupozen(width, ff, layers, heads, q_rank, vocab, window, experts=None):
    stack, mixer = [], _latent_mixer(heads, q_rank, window)
    for i in range(layers):
        if experts and i % 2:
            n, size, top = experts
            stack.append({"type": "latent_attention", "mixer": {**mixer, "kv_from": i - 1},
                          "mlp": {"kind": "moe", "expert": {"ff": size}, "router": {"experts": n, "top": top}}})
        else:
            stack.append({"type": "latent_attention", "mixer": mixer, "mlp": {"kind": "dense", "ff": ff}})
    return {"architecture": "Bupozen", "layers": stack, "norm": {"eps": 1e-5}, "vocab": vocab, "width": width}


# the language models of the benchmark that the cases use
MODELS = {
    "w3072_l26": _kegizen(3072, 9216, 26, 24, 8, 32, 8, 8320, 1024),
    "w2048_l16_loop": _kegizen(2048, 5632, 16, 16, 8, 16, 4, 32768, 512, (4, 12, 2)),
    "latent_w3072_l26": _bupozen(3072, 13824, 26, 32, 1536, 8320, 1024),
    "latent_w2048_l16_experts": _bupozen(2048, 8448, 16, 16, 768, 32768, 512, (64, 1024, 6)),
}


def listed():
    return [
        # the smallest call: a chunk of a stream, 0.4 s of audio at once
        {"name": "codec_chunk", "kind": "codec", "frames": 5},
        # a whole text's waveform: 49 s of audio
        {"name": "codec_utterance", "kind": "codec", "frames": 611},
        # time to the first audio frame after a short text with a short voice sample
        {"name": "first_frame", "kind": "prompt", "voice": 40, "text": 13, "frames": 1},
        # the same with a long voice sample and a paragraph of text, and some frames one host call each
        {"name": "long_prompt", "kind": "prompt", "voice": 903, "text": 295, "frames": 3},
        # the benchmark's utterance: 256 prompt rows, 17 s of audio, the frame loop on the device
        {"name": "utterance", "kind": "utterance", "prompt": 256, "frames": 212},
        # eight callers served in lock step, prompts of uneven lengths
        {"name": "batch", "kind": "batch", "utterances": 8, "prompt": 187, "frames": 24},
        # the reference's own orchestration of a frame: prefill, then one decoder step and 14 velocity calls per frame
        {"name": "reference_calls", "kind": "calls", "prompt": 41, "frames": 2},
        # reading a long document with delta-rule and windowed layers
        {"name": "lm_prompt", "kind": "lm", "model": "w3072_l26", "dtype": "bfloat16", "prompt": 4001, "new": 0, "portion": 0},
        # an answer to a chat turn, chosen greedily on the device
        {"name": "lm_answer", "kind": "lm", "model": "w3072_l26", "dtype": "bfloat16", "prompt": 203, "new": 32, "portion": 0},
        # a long document with latent attention
        {"name": "latent_prompt", "kind": "lm", "model": "latent_w3072_l26", "dtype": "bfloat16", "prompt": 2500, "new": 0, "portion": 0},
        # a mixture of experts: a chat turn, then a program that samples each token itself
        {"name": "experts_sampling", "kind": "lm", "model": "latent_w2048_l16_experts", "dtype": "bfloat16", "prompt": 331, "new": 40, "portion": 1},
        # 32-bit products throughout: a prompt, then drafted tokens checked five at a time, with a looped stack
        {"name": "loop_float32", "kind": "lm", "model": "w2048_l16_loop", "dtype": "float32", "prompt": 390, "new": 15, "portion": 5},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(["codec", "prompt", "utterance", "batch", "calls", "lm", "lm", "lm"])
    if kind == "codec":
        return {"kind": kind, "frames": spread(1, 620)}
    if kind == "prompt":
        return {"kind": kind, "voice": spread(10, 900), "text": spread(3, 290), "frames": rng.randint(1, 3)}
    if kind == "utterance":
        return {"kind": kind, "prompt": spread(16, 600), "frames": spread(4, 150)}
    if kind == "batch":
        return {"kind": kind, "utterances": rng.randint(2, 8), "prompt": spread(20, 250), "frames": spread(2, 24)}
    if kind == "calls":
        return {"kind": kind, "prompt": spread(8, 300), "frames": rng.randint(1, 3)}
    model = rng.choice(sorted(MODELS))
    if model == "w2048_l16_loop" and rng.random() < 0.4:
        return {"kind": kind, "model": model, "dtype": "float32", "prompt": spread(30, 400), "new": rng.randint(0, 12), "portion": rng.randint(1, 6)}
    how = rng.choice(["read", "greedy", "portions"])
    return {"kind": kind, "model": model, "dtype": "bfloat16", "prompt": spread(20, 4000),
            "new": 0 if how == "read" else spread(4, 32), "portion": rng.choice([1, 1, 2, 5, 9, 17]) if how == "portions" else 0}


# ---------------------------------------------------------------------------------------------- models

_kept = {}


def _once(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def _speech_weights():
    """Random weights of the speech model. The semantic head never says END, so that an utterance has its case's
    length. The rows of the acoustic codes are small beside the semantic ones: a latent that lies on the boundary
    between two codes, where the order of a sum decides, then hardly steers the frames after it."""
    def make():
        pkg = package()
        m = pkg.SynthModel(seed=1234, semantic_bias=True)
        m.t["acoustic_transformer.semantic_codebook_output.bias"][1] = -1000.0
        table = m.t["mm_audio_embeddings.audio_codebook_embeddings.embeddings.weight"]
        wide = (table[8194:].astype(np.uint32) << 16).view(np.float32) * np.float32(2.0 ** -18)   # exact in BF16
        table[8194:] = (wide.view(np.uint32) >> 16).astype(np.uint16)
        return m
    return _once("speech weights", make)


def _codec_weights():
    return _once("codec weights", lambda: package().SynthCodec(seed=77))


def _engine():
    return _once("engine", lambda: package().Engine(kv_cache_max=KV_ROWS))


def _speech():
    def make():
        _engine().upload(_speech_weights(), decoder=True, acoustic=True, audio_table=True, token_table=True)
        return True
    _once("speech", make)
    return _engine()


def _codec():
    _once("codec", lambda: _engine().codec_upload(_codec_weights()) or True)
    return _engine()


def _language_model(name, dtype):
    return _once((name, dtype), lambda: package().LanguageModel(config=MODELS[name], dtype=dtype, max_tokens=LM_TOKENS, seed=7))


# ---------------------------------------------------------------------------------------------- inputs

def _inputs(case, seed):
    """Host arrays: what the entry points take."""
    rng = np.random.default_rng([int(seed), 20])
    kind = case["kind"]
    if kind == "codec":
        n = case["frames"]
        return {"codes": np.concatenate([rng.integers(2, 8194, (n, 1)), rng.integers(2, 23, (n, 36))], axis=1).astype(np.int32)}
    if kind == "lm":
        vocab = MODELS[case["model"]]["vocab"]
        return {"prompt": rng.integers(0, vocab, case["prompt"]).astype(np.int32), "next": rng.integers(0, vocab, case["new"]).astype(np.int32)}

    def rows(n, sigma=0.5):                 # voice rows, or rows of both kinds
        return (rng.standard_normal((n, 3072), dtype=np.float32) * np.float32(sigma)).astype(np.float32)

    f = case["frames"]
    if kind == "prompt":
        voice = rows(case["voice"]).view(np.uint32) >> 16
        return {"voice": voice.astype(np.uint16), "ids": rng.integers(1000, 131072, case["text"]).astype(np.int32),
                "embeds": rows(f, 0.02), "noise": rng.standard_normal((f, 36), dtype=np.float32)}
    if kind == "utterance":
        return {"rows": rows(case["prompt"]), "first": rows(1, 0.02)[0], "noise": rng.standard_normal((f, 36), dtype=np.float32)}
    if kind == "batch":
        n = case["utterances"]
        lengths = [max(1, case["prompt"] - (u * 29) % max(2, case["prompt"] // 2)) for u in range(n)]
        return {"prompts": [rows(r) for r in lengths], "firsts": rows(n, 0.02), "noise": rng.standard_normal((n, f, 36), dtype=np.float32)}
    return {"rows": rows(case["prompt"]), "embeds": rows(f, 0.02), "noise": rng.standard_normal((f, 36), dtype=np.float32)}


def prepare(case, seed):
    s = {"case": case, **_inputs(case, seed)}
    if case["kind"] == "codec":
        s["engine"] = _codec()
    elif case["kind"] == "lm":
        s["lm"] = _language_model(case["model"], case["dtype"])
    else:
        s["engine"] = _speech()
    return s


# ---------------------------------------------------------------------------------------------- one pass

TIMES = np.linspace(0.0, 1.0, 8, dtype=np.float32)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "codec":
        return s["engine"].codec_decode(s["codes"])[0]
    if kind == "lm":
        return _run_lm(s, case)
    eng = s["engine"]
    if kind == "prompt":
        pos = eng.prefill_prompt(s["ids"], s["voice"])
        codes, hidden = [], []
        for f in range(case["frames"]):     # the program makes the next input row itself
            c, h = eng.frame(s["embeds"][f], s["noise"][f], pos + f)
            codes.append(c)
            hidden.append(h)
        return {"codes": np.stack(codes), "hidden": np.stack(hidden)}
    if kind == "utterance":
        eng.prefill(s["rows"])
        return {"codes": eng.utterance(s["first"], case["prompt"], s["noise"])[0]}
    if kind == "batch":
        codes, _, hidden, _ = eng.batch(s["prompts"], s["firsts"], s["noise"])
        return {"codes": np.stack(codes), "hidden": hidden}
    eng.prefill(s["rows"])
    hidden, latents = [], []
    nothing = np.zeros(3072, dtype=np.float32)
    for f in range(case["frames"]):
        h = eng.llm_forward(s["embeds"][f], case["prompt"] + f)
        x = s["noise"][f].copy()
        for t, u in zip(TIMES[:-1], TIMES[1:]):
            with_text, without = eng.predict_velocity(x, h, t), eng.predict_velocity(x, nothing, t)
            x = x + (np.float32(1.2) * with_text + (np.float32(1.0) - np.float32(1.2)) * without) * (u - t)
        hidden.append(h)
        latents.append(x)
    return {"hidden": np.stack(hidden), "latents": np.stack(latents)}


def _run_lm(s, case):
    lm = s["lm"]
    seq = lm.open()
    try:
        if case["new"] == 0:
            return {"logits": lm.step(seq, s["prompt"], want=[-1])}
        if case["portion"] == 0:
            tokens = lm.generate(seq, s["prompt"], case["new"])
            return {"tokens": np.array(tokens, dtype=np.int32), "logits": lm.step(seq, tokens[-1:], want=[0])}
        out, p = [lm.step(seq, s["prompt"], want=[-1])], case["portion"]
        for i in range(0, case["new"], p):
            t = s["next"][i:i + p]
            out.append(lm.step(seq, t, want=range(len(t))))
        return {"logits": np.concatenate(out)}
    finally:
        lm.release(seq)


# ---------------------------------------------------------------------------------------------- what a pass cannot do without

LAYER = 2 * (6144 * 3072 + 3072 * 4096 + 3 * 9216 * 3072)      # bytes of a speech layer's matrices
DECODER, ACOUSTIC = 26 * LAYER, 3 * LAYER
HEADS = 2 * (8320 + 3072) * 3072                               # semantic head, hidden-state projection


def _frame_work(keys, batch=1):
    """Weights are read once per frame for all utterances, the acoustic ones once per step of the flow."""
    small = 2 * 2 * 36 * 3072
    b = DECODER + HEADS + 7 * (ACOUSTIC + small) + batch * 26 * keys * 8192
    return b, batch * (DECODER + HEADS + 7 * 6 * ACOUSTIC + 26 * keys * 4 * 4096)


def _prefill_work(n):
    return DECODER + 26 * n * 8192 + 4 * n * 3072, n * DECODER + 26 * 4 * 4096 * n * (n + 1) // 2


def _lm_layers(c):
    """(matrix elements that a token uses, elements read when many tokens pass, attention operations and cached bytes per key, window)"""
    n, loop = len(c["layers"]), c.get("loop")
    order = list(range(n))
    if loop:
        order = list(range(loop["start"])) + list(range(loop["start"], loop["stop"])) * loop["times"] + list(range(loop["stop"], n))
    w = c["width"]
    out = []
    for i in order:
        spec = c["layers"][i]
        m, mlp = spec["mixer"], spec["mlp"]
        h, d, v = m["heads"], m["dim"], m["vdim"]
        if spec["type"] == "delta":
            g = m["kv_heads"]
            e, per_key, cached, window, state = w * (2 * g * d + 2 * h * v + 2 * h) + w * h * v, 0, 0, 0, h * d * v
        elif spec["type"] == "attention":
            g = m["kv_heads"]
            e, per_key, cached, window, state = w * (h * d + g * (d + v)) + w * h * v, 2 * h * (d + v), 4 * g * (d + v), m["mask"]["size"], 0
        else:
            r, q, x = m["kv_rank"], m["q_rank"], m["rot_dim"]
            e = w * q + (0 if m.get("kv_from") is not None else w * (r + x)) + w * h + q * h * (d + x) + r * h * (d + v) + w * h * v
            per_key, cached, window, state = 2 * h * (d + x + v), 4 * (r + x), m["mask"]["size"], 0
        used = read = e
        if mlp["kind"] == "moe":
            one, top, many = 2 * w * mlp["expert"]["ff"], mlp["router"]["top"], mlp["router"]["experts"]
            used, read = e + top * one + many * w, e + many * one + many * w
        else:
            ff = (3 if c["architecture"] == "Kegizen" else 2) * w * mlp["ff"]
            used, read = e + ff, e + ff
        out.append((used, read, per_key, cached, window, state))
    return out


def _lm_work(case):
    c = MODELS[case["model"]]
    layers, head = _lm_layers(c), c["vocab"] * c["width"]
    size = 2
    portions = [case["prompt"]]
    if case["new"]:
        p = max(1, case["portion"])
        portions += [min(p, case["new"] - i) for i in range(0, case["new"], p)]
    b = f = at = 0
    for k, n in enumerate(portions):
        wanted = 1 if k == 0 else n
        b += size * head + 4 * wanted * c["vocab"] + size * n * c["width"]
        f += 2 * wanted * head
        for used, read, per_key, cached, window, state in layers:
            moe = read - used
            b += size * (used + (moe if n >= 32 else 0)) + 8 * state
            keys = sum(min(at + i + 1, window) for i in range(n)) if window else 0
            f += 2 * used * n + per_key * keys + 6 * state * n
            b += cached * (min(at, window) + n)
        at += n
    return b, f


def work(case):
    kind = case["kind"]
    if kind == "codec":
        n = case["frames"]
        rows = 2 * (n + 2 * n + 4 * n + 8 * n)                    # two layers at each rate
        layer = 4 * 1024 * 1024 + 3 * 4096 * 1024
        conv = [1024 * 292 * 3, 2 * 1024 * 1024 * 2, 2 * 1024 * 1024 * 2, 2 * 1024 * 1024 * 2, 240 * 1024 * 7]
        times = [n, n, 2 * n, 4 * n, 8 * n]
        return {"bytes": 2 * 8 * layer + 4 * sum(conv) + 37 * 4 * n + 1024 * n + 4 * 1920 * n,
                "flops": 2 * rows * layer + 2 * sum(a * b for a, b in zip(conv, times))}
    if kind == "lm":
        b, f = _lm_work(case)
        return {"bytes": b, "flops": f}
    parts = []
    if kind == "batch":
        n = case["utterances"]
        lengths = [max(1, case["prompt"] - (u * 29) % max(2, case["prompt"] // 2)) for u in range(n)]
        parts += [_prefill_work(r) for r in lengths]
        parts += [_frame_work(sum(lengths) // n + i + 1, n) for i in range(case["frames"])]
    else:
        n = case["voice"] + case["text"] + 5 if kind == "prompt" else case["prompt"]
        parts.append(_prefill_work(n))
        parts += [_frame_work(n + i + 1) for i in range(case["frames"])]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """About four times what the cases were seen to be off exact() by, the largest over several seeds."""
    kind = case["kind"]
    if kind == "codec":                       # 2.1e-5
        return {"rel": 8e-5}
    if kind == "utterance":                   # a code whose latent lies on a boundary may fall on either side
        return {"differ": 0.01}
    if kind == "lm":
        if case["dtype"] == "float32":        # 5.5e-6
            return {"rel": 2e-5}
        if case["model"] == "latent_w2048_l16_experts":   # 4.3e-6; a token whose experts nearly tie may go to another one
            return {"rel": 1e-3}
        return {"rel": 4e-4, "differ": 0.0}   # 8.6e-5
    return {"rel": 2e-4, "differ": 0.01}      # hidden states 4.6e-5


# ---------------------------------------------------------------------------------------------- the same in 64 bits

F64 = torch.float64
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def _dev(a, dtype=F64):
    return torch.as_tensor(np.asarray(a)).to(DEVICE).to(dtype)


def _bf16_host(a):
    """A host array of BF16 patterns, on the device."""
    return _once(("weight", a.ctypes.data), lambda: torch.from_numpy(a.view(np.int16)).to(DEVICE).view(torch.bfloat16))


def _silu(z):
    return z * torch.sigmoid(z)


def _rms(x, gain, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _centred(x, gain, eps):
    d = x - x.mean(-1, keepdim=True)
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * gain


def _attend(q, k, v, scale, cap, visible):
    """q [T, H, d], k [S, G, d], v [S, G, e], visible [T, S] -> [T, H, e]; one head at a time."""
    share = q.shape[1] // k.shape[1]
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=F64, device=q.device)
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // share].T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        out[:, h] = torch.softmax(s.masked_fill(~visible, -math.inf), dim=1) @ v[:, h // share]
    return out


class _ExactSpeech:
    """The speech model: decoder layers with a cache, the flow of a frame."""

    def __init__(self):
        self.t = _speech_weights().t
        self.k, self.v = [None] * 26, [None] * 26

    def mat(self, name):
        return _bf16_host(self.t[name + ".weight"]).double()

    def gain(self, name):
        return _dev(self.t[name + ".weight"])

    def layer(self, x, name, attend):
        h = _rms(x, self.gain(name + ".attention_norm"), 1e-5)
        q, k, v = (h @ self.mat(f"{name}.attention.w{c}").T for c in "qkv")
        x = x + attend(q, k, v) @ self.mat(name + ".attention.wo").T
        h = _rms(x, self.gain(name + ".ffn_norm"), 1e-5)
        return x + (_silu(h @ self.mat(name + ".feed_forward.w1").T) * (h @ self.mat(name + ".feed_forward.w3").T)) @ self.mat(name + ".feed_forward.w2").T

    def decode(self, x):
        """The next rows of the sequence [n, 3072]; their outputs."""
        for l in range(26):
            def attend(q, k, v, l=l):
                n, at = q.shape[0], 0 if self.k[l] is None else self.k[l].shape[0]
                # angles are those of 32-bit frequencies, as the reference defines them
                f = np.float32(1.0) / np.power(np.float32(1e6), np.arange(0, 128, 2, dtype=np.float32) / np.float32(128))
                a = _dev((np.arange(at, at + n, dtype=np.float32)[:, None] * f[None]).astype(np.float32))
                c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]

                def turn(y):
                    y = y.view(n, -1, 64, 2)
                    return torch.stack([y[..., 0] * c - y[..., 1] * s, y[..., 0] * s + y[..., 1] * c], -1).view(n, -1, 128)
                k, v = turn(k), v.view(n, 8, 128)
                self.k[l] = k if at == 0 else torch.cat([self.k[l], k])
                self.v[l] = v if at == 0 else torch.cat([self.v[l], v])
                seen = torch.arange(at + n, device=x.device)[None] <= torch.arange(at, at + n, device=x.device)[:, None]
                return _attend(turn(q), self.k[l], self.v[l], 128 ** -0.5, 0, seen).reshape(n, 4096)
            x = self.layer(x, f"layers.{l}", attend)
        return _rms(x, self.gain("norm"), 1e-5)

    def velocity(self, x, hidden, t):
        """x [n, 36], hidden [n, 3072]: n independent passes of three tokens."""
        p, n = "acoustic_transformer", x.shape[0]
        a = np.float32(t) * self.t[f"{p}.time_embedding.inv_freq"]
        e = _dev(np.concatenate([np.cos(a), np.sin(a)])) @ self.mat(f"{p}.time_projection").T
        y = torch.stack([x @ self.mat(f"{p}.input_projection").T, e.expand(n, -1), hidden @ self.mat(f"{p}.llm_projection").T], 1)

        def attend(q, k, v):
            q, k, v = q.view(n, 3, 8, 4, 128), k.view(n, 3, 8, 128), v.view(n, 3, 8, 128)
            s = torch.softmax(torch.einsum("nigrd,njgd->ngrij", q, k) * 128 ** -0.5, -1)
            return torch.einsum("ngrij,njgd->nigrd", s, v).reshape(n, 3, 4096)
        for l in range(3):
            y = self.layer(y, f"{p}.layers.{l}", attend)
        return _rms(y[:, 0], self.gain(f"{p}.norm"), 1e-5) @ self.mat(f"{p}.acoustic_codebook_output").T

    def flow(self, hidden, noise):
        x, both = noise[None], torch.stack([hidden, torch.zeros_like(hidden)])
        for t, u in zip(TIMES[:-1], TIMES[1:]):
            v = self.velocity(x.expand(2, -1), both, t)
            x = x + (1.2 * v[0] - 0.2 * v[1])[None] * float(u - t)
        return x[0]

    def codes(self, hidden, noise):
        p = "acoustic_transformer.semantic_codebook_output"
        z = hidden @ self.mat(p).T + _dev(self.t[p + ".bias"])
        z[0] = -1e30
        z[8194:] = -1e30
        level = torch.floor((self.flow(hidden, noise).clamp(-1, 1) + 1) / 2 * 20 + 0.5).clamp(0, 20)
        return [int(z.argmax())] + [int(i) + 2 for i in level]

    def embed(self, codes):
        table = _bf16_host(self.t["mm_audio_embeddings.audio_codebook_embeddings.embeddings.weight"])
        rows = [codes[0]] + [8194 + 23 * i + c for i, c in enumerate(codes[1:])]
        return table[rows].double().sum(0)


def _exact_speech(case, s):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for u, rows in enumerate(s["prompts"]):
            m, e = _ExactSpeech(), _dev(s["firsts"][u])
            m.decode(_dev(rows))
            for f in range(case["frames"]):
                h = m.decode(e[None])[0]
                if f + 1 < case["frames"]:
                    e = m.embed(m.codes(h, _dev(s["noise"][u, f])))
            out.append(h)
        return {"codes": None, "hidden": torch.stack(out)}
    m = _ExactSpeech()
    if kind == "prompt":
        model = _speech_weights()
        ids = [[1], [25], [36], list(s["ids"]), [35], [25]]
        text = [_dev(model.token_rows(i)) for i in ids]
        voice = _dev((s["voice"].astype(np.uint32) << 16).view(np.float32))
        m.decode(torch.cat([text[0], text[1], voice, *text[2:]]))
        return {"codes": None, "hidden": torch.stack([m.decode(_dev(e)[None])[0] for e in s["embeds"]])}
    m.decode(_dev(s["rows"]))
    hidden = [m.decode(_dev(e)[None])[0] for e in s["embeds"]]
    return {"hidden": torch.stack(hidden), "latents": torch.stack([m.flow(h, _dev(z)) for h, z in zip(hidden, s["noise"])])}


def _exact_codec(s):
    w = _codec_weights().t
    codes = torch.as_tensor(s["codes"]).to(DEVICE).long()
    x = torch.cat([_dev(w["semantic_embedding"])[(codes[:, 0] - 2).clamp(0, 8191)],
                   (codes[:, 1:] - 2).clamp(0, 20).double() / 10.0 - 1.0], 1)

    def conv(x, name):
        """Causal, with the reference's rule at the left end: a place before the first row is mirrored, or nothing."""
        a, n = _dev(w[f"{name}.weight"]), x.shape[0]
        y = _dev(w[f"{name}.bias"]).expand(n, -1)
        for tap in range(a.shape[2]):
            src = (torch.arange(n, device=x.device) + tap - (a.shape[2] - 1)).abs()
            y = y + (x[src.clamp(max=n - 1)] * (src < n)[:, None]) @ a[:, :, tap].T
        return y

    x = conv(x, "input_conv")
    for l in range(8):
        n, T, window = f"codec.layers.{l}", x.shape[0], (2, 4, 8, 16)[l // 2]
        h = _rms(x, _dev(w[f"{n}.attention_norm"]), 1e-2)
        q, k, v = (h @ _dev(w[f"{n}.w{c}"]).T for c in "qkv")
        q, k = _rms(q, _dev(w[f"{n}.q_norm"]), 1e-6), _rms(k, _dev(w[f"{n}.k_norm"]), 1e-6)
        q, k, v = (a.view(T, 8, 128) for a in (q, k, v))
        back = torch.arange(window, device=x.device)
        src = torch.arange(T, device=x.device)[:, None] - back[None]                  # [T, window]
        score = torch.einsum("thd,twhd->twh", q, k[src.clamp(min=0)]) * 128 ** -0.5
        score = score - _dev([2.0 ** -(i + 1) for i in range(8)])[None, None] * back[None, :, None]
        p = torch.softmax(score.masked_fill((src < 0)[:, :, None], -math.inf), 1)
        y = torch.einsum("twh,twhd->thd", p, v[src.clamp(min=0)]).reshape(T, 1024) @ _dev(w[f"{n}.wo"]).T
        x = x + y * _dev(w[f"{n}.attn_scale"])
        h = _rms(x, _dev(w[f"{n}.ffn_norm"]), 1e-2)
        x = x + ((_silu(h @ _dev(w[f"{n}.w1"]).T) * (h @ _dev(w[f"{n}.w3"]).T)) @ _dev(w[f"{n}.w2"]).T) * _dev(w[f"{n}.ffn_scale"])
        if l in (1, 3, 5):
            a, b = _dev(w[f"up{l // 2}.weight"]), _dev(w[f"up{l // 2}.bias"])
            before = torch.cat([torch.zeros_like(x[:1]), x[:-1]])
            x = torch.stack([x @ a[:, :, i] + before @ a[:, :, i + 2] + b for i in (0, 1)], 1).reshape(2 * T, 1024)
    return conv(x, "output_proj").reshape(-1)


def _hash_name(name, seed):
    h = 2166136261 ^ seed
    for c in name.encode():
        h = (h ^ c) * 16777619 & 0xFFFFFFFF
    return h


def _hashed_matrix(name, shape, seed):
    """A matrix of a model with random weights: BF16 values, about N(0, 0.02^2)."""
    n, m32 = shape[0] * shape[1], 0xFFFFFFFF
    out = torch.empty(n, dtype=torch.bfloat16, device=DEVICE)
    for a in range(0, n, 1 << 25):
        i = torch.arange(a, min(n, a + (1 << 25)), device=DEVICE, dtype=torch.int64)
        h = (i * 2654435761 & m32) ^ ((i >> 32) * 40503) ^ _hash_name(name, seed)
        s = torch.zeros(i.shape, dtype=torch.float32, device=DEVICE)
        for _ in range(4):
            h ^= h >> 16
            h = h * 0x7FEB352D & m32
            h ^= h >> 15
            h = h * 0x846CA68B & m32
            h ^= h >> 16
            s += (h >> 8).float() * 2.0 ** -24 - 0.5
        out[a:a + i.numel()] = s * float(np.float32(0.02) * np.float32(1.7320508))
    return out.view(shape)


def _hashed_vector(name, n, seed):
    """Gains 1 + N(0, 0.02^2), logarithms of decays N(0, 0.5^2), others N(0, 0.3^2)."""
    h, out = _hash_name(name, seed), []
    for _ in range(n):
        s = -2.0
        for _ in range(4):
            h = (h * 1664525 + 1013904223) & 0xFFFFFFFF
            s += (h >> 8) / 16777216.0
        out.append(s)
    out = np.array(out, dtype=np.float32) * np.float32(1.7320508)
    if "norm" in name:
        return np.float32(1.0) + np.float32(0.02) * out
    return np.float32(0.5 if "A_log" in name else 0.3) * out


class _ExactLm:
    """A language model over the tokens of one sequence, portion by portion."""

    def __init__(self, name, seed=7):
        self.name, self.c, self.seed = name, MODELS[name], seed
        self.mem, self.at = {}, 0

    def mat(self, name, *shape):
        return _once((self.name, name), lambda: _hashed_matrix(name, shape, self.seed)).double()

    def vec(self, name, n):
        return _once((self.name, name), lambda: _dev(_hashed_vector(name, n, self.seed)))

    def kept(self, key, new):
        old = self.mem.get(key)
        self.mem[key] = new if old is None else torch.cat([old, new])
        return self.mem[key]

    def angles(self, rot, n):
        d, base = rot["dims"], rot["base"]
        i = np.arange(d // 2, dtype=np.float64)
        f, mag, sc = base ** (-2.0 * i / d), 1.0, rot.get("scaling")
        if sc:
            def turn(t):
                return d * math.log(sc["original"] / (2.0 * math.pi * t)) / (2.0 * math.log(base))
            lo, hi = max(math.floor(turn(sc["fast"])), 0), min(math.ceil(turn(sc["slow"])), d - 1)
            r = np.clip((i - lo) / max(hi - lo, 0.001), 0.0, 1.0)
            f, mag = f / sc["factor"] * r + f * (1.0 - r), 0.1 * math.log(sc["factor"]) + 1.0
        a = torch.arange(self.at, self.at + n, dtype=F64, device=DEVICE)[:, None, None] * _dev(f)
        return torch.cos(a) * mag, torch.sin(a) * mag

    def visible(self, n, mask):
        i = torch.arange(self.at, self.at + n, device=DEVICE)[:, None]
        j = torch.arange(self.at + n, device=DEVICE)[None]
        return (j <= i) & ((i - j < mask["size"]) | (j < mask.get("keep_first", 0)))

    def attention(self, h, p, m, key):
        n, w = h.shape
        H, G, d, e = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        eps, half = self.c["norm"]["eps"], m["rot"]["dims"] // 2
        c, s = self.angles(m["rot"], n)

        def turn(x):
            u, v = x[..., :half], x[..., half:2 * half]
            return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)
        q = turn(_rms(h @ self.mat(p + ".q", H * d, w).T, self.vec(p + ".q.norm", H * d), eps).view(n, H, d))
        k = turn(_rms(h @ self.mat(p + ".k", G * d, w).T, self.vec(p + ".k.norm", G * d), eps).view(n, G, d))
        k, v = self.kept((key, "k"), k), self.kept((key, "v"), (h @ self.mat(p + ".v", G * e, w).T).view(n, G, e))
        return _attend(q, k, v, m["scale"], m.get("softcap"), self.visible(n, m["mask"])).reshape(n, H * e) @ self.mat(p + ".o", w, H * e).T

    def delta(self, h, p, m, key):
        n, w = h.shape
        H, G, d, e, taps = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["conv"]
        parts = []
        for name, rows in (("q", G * d), ("k", G * d), ("v", H * e)):
            x = h @ self.mat(f"{p}.{name}", rows, w).T
            old = self.mem.get((key, name))
            x = torch.cat([torch.zeros((taps - 1, rows), dtype=F64, device=DEVICE) if old is None else old, x])
            self.mem[(key, name)] = x[-(taps - 1):]
            a = self.vec(f"{p}.{name}.conv", rows * taps).view(rows, taps)
            parts.append(_silu(sum(x[j:j + n] * a[:, j] for j in range(taps))))
        q, k, v = parts[0].view(n, G, d), parts[1].view(n, G, d), parts[2].view(n, H, e)
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
        beta = torch.sigmoid(h @ self.mat(p + ".b", H, w).T)
        soft = torch.nn.functional.softplus(h @ self.mat(p + ".a", H, w).T + self.vec(p + ".dt_bias", H), threshold=200)
        decay = torch.exp(-torch.exp(self.vec(p + ".A_log", H)) * soft)
        state = self.mem.get((key, "s"))
        state = torch.zeros((H, d, e), dtype=F64, device=DEVICE) if state is None else state
        out = torch.empty((n, H, 1, e), dtype=F64, device=DEVICE)
        qr, kr, kc, vr = q[:, :, None], k[:, :, None], k[..., None], v[:, :, None]
        g, b = decay[..., None, None], beta[..., None, None]
        for t in range(n):
            state = state * g[t]
            state = torch.baddbmm(state, kc[t], (vr[t] - torch.bmm(kr[t], state)) * b[t])
            torch.bmm(qr[t], state, out=out[t])
        self.mem[(key, "s")] = state
        gate = _silu(h @ self.mat(p + ".g", H * e, w).T).view(n, H, e)
        y = _rms(out[:, :, 0], self.vec(p + ".norm", e), self.c["norm"]["eps"]) * gate
        return y.reshape(n, H * e) @ self.mat(p + ".o", w, H * e).T

    def latent(self, h, p, m, i):
        n, w = h.shape
        H, d, x, e, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
        eps = self.c["norm"]["eps"]
        c, s = self.angles(m["rot"], n)

        def turn(y):
            u, v = y[..., 0::2], y[..., 1::2]
            return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
        if m.get("kv_from") is None:
            y = h @ self.mat(p + ".dkv", r + x, w).T
            self.kept((i, "c"), _rms(y[:, :r], self.vec(p + ".dkv.norm", r), eps))
            self.kept((i, "x"), turn(y[:, None, r:]))
            src = i
        else:
            src = m["kv_from"]
        latents, shared = self.mem[(src, "c")], self.mem[(src, "x")]
        q = _rms(h @ self.mat(p + ".dq", m["q_rank"], w).T, self.vec(p + ".dq.norm", m["q_rank"]), eps)
        q = (q @ self.mat(p + ".uq", H * (d + x), m["q_rank"]).T).view(n, H, d + x)
        q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
        S = latents.shape[0]
        k = torch.cat([(latents @ self.mat(p + ".uk", H * d, r).T).view(S, H, d), shared.expand(-1, H, -1)], -1)
        v = (latents @ self.mat(p + ".uv", H * e, r).T).view(S, H, e)
        gate = torch.sigmoid(h @ self.mat(p + ".g", H, w).T)
        out = _attend(q, k, v, m["scale"], 0, self.visible(n, m["mask"])) * gate[..., None]
        return out.reshape(n, H * e) @ self.mat(p + ".o", w, H * e).T

    def experts(self, h, p, spec):
        w, ff, top, many = h.shape[1], spec["expert"]["ff"], spec["router"]["top"], spec["router"]["experts"]
        z, chosen = torch.topk(h @ self.mat(p + ".router", many, w).T, top, dim=1)
        weight, y = torch.softmax(z, 1), torch.zeros_like(h)
        for e in range(many):
            rows, slot = torch.nonzero(chosen == e, as_tuple=True)
            if rows.numel():
                a = torch.relu(h[rows] @ self.mat(f"{p}.e{e}.up", ff, w).T) ** 2 @ self.mat(f"{p}.e{e}.down", w, ff).T
                y[rows] += weight[rows, slot][:, None] * a
        return y

    def layer(self, x, i, key):
        spec, eps, w, p = self.c["layers"][i], self.c["norm"]["eps"], self.c["width"], f"l{i}"
        mlp = spec["mlp"]
        if self.c["architecture"] == "Bupozen":
            h = _rms(x, self.vec(p + ".norm1", w), eps)
            y = self.latent(h, p + ".mix", spec["mixer"], i)
            if mlp["kind"] == "moe":
                return x + y + self.experts(h, p + ".mlp", mlp)
            return x + y + torch.relu(h @ self.mat(p + ".mlp.up", mlp["ff"], w).T) ** 2 @ self.mat(p + ".mlp.down", w, mlp["ff"]).T
        mixer = self.delta if spec["type"] == "delta" else self.attention
        h = mixer(_centred(x, self.vec(p + ".norm1", w), eps), p + ".mix", spec["mixer"], key)
        x = x + _centred(h, self.vec(p + ".norm1b", w), eps)
        h = _centred(x, self.vec(p + ".norm2", w), eps)
        y = _silu(h @ self.mat(p + ".mlp.gate", mlp["ff"], w).T) * (h @ self.mat(p + ".mlp.up", mlp["ff"], w).T)
        return x + _centred(y @ self.mat(p + ".mlp.down", w, mlp["ff"]).T, self.vec(p + ".norm2b", w), eps)

    def feed(self, tokens, wanted):
        """The next tokens; the logits at the wanted places."""
        w, vocab, loop = self.c["width"], self.c["vocab"], self.c.get("loop")
        n = len(self.c["layers"])
        first = x = self.mat("embed", vocab, w)[torch.as_tensor(np.asarray(tokens)).to(DEVICE).long()]
        runs = [(i, False) for i in range(loop["start"] if loop else n)]
        if loop:
            runs += [(i, i == loop["start"]) for _ in range(loop["times"]) for i in range(loop["start"], loop["stop"])]
            runs += [(i, False) for i in range(loop["stop"], n)]
        for r, (i, begins) in enumerate(runs):
            if begins:
                x = torch.cat([x, first], 1) @ self.mat("loop.in", w, 2 * w).T
            x = self.layer(x, i, r)
        self.at += len(tokens)
        norm = _rms if self.c["architecture"] == "Bupozen" else _centred
        return norm(x[wanted], self.vec("final.norm", w), self.c["norm"]["eps"]) @ self.mat("head", vocab, w).T


def exact(case, seed):
    s, kind = _inputs(case, seed), case["kind"]
    with torch.no_grad():
        if kind == "utterance":               # whole numbers alone
            return None
        if kind == "codec":
            return _exact_codec(s)
        if kind != "lm":
            return _exact_speech(case, s)
        m = _ExactLm(case["model"])
        out = [m.feed(s["prompt"], [len(s["prompt"]) - 1])]
        if case["new"] and case["portion"] == 0:
            for _ in range(case["new"]):
                out = [m.feed([int(out[0][0].argmax())], [0])]
            return {"tokens": None, "logits": out[0]}
        for i in range(0, case["new"], max(1, case["portion"])):
            t = s["next"][i:i + case["portion"]]
            out.append(m.feed(t, list(range(len(t)))))
        return {"logits": torch.cat(out)}
