"""What users of this library have it do, as measurable cases.

Three ways in, each through the package's public entry points:

* a buffer already in device memory (``Session.apply_device_async`` and ``device_result``): the
  replace step of a program whose data lives on the GPU;
* host bytes to host bytes: one-shot ``unified``, a session that takes a document through a chain
  of pairs (``reset``, ``apply_batch``, ``result``), and ``gpu_replace_streaming``;
* many independent documents, each with its own pairs (``replace_jobs``).

Inputs have the shapes of ``cuda_replace_b200.workloads``: Zipf text with HTML-entity-like tokens,
ACGT sequences, uniform random bytes, runs of one byte, and text with rule lines. They are made
on the GPU from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from cuda_replace_b200 import workloads as W
from cuda_replace_b200.cuda_replace_wrapper import (CudaReplaceLib, Session, gpu_replace_streaming,
                                                    replace_jobs)

KiB, MiB, GiB = 1 << 10, 1 << 20, 1 << 30


# ------------------------------------------------------------------ the cases
def listed() -> list:
    return [
        # one web page in device memory, one entity unescaped: launch and read-back latency
        dict(name="page_entity", path="device", data="text", n=48 * KiB + 13, pat="&tok0;", rep="&"),
        # a 16 MiB sequence, one motif masked: the library's smallest benchmark input
        dict(name="acgt_motif", path="device", data="acgt", n=16 * MiB, pat="ACGT", rep="N"),
        # URL-escaping the blanks of a text: a match every few bytes, each growing
        dict(name="text_blanks", path="device", data="text", n=64 * MiB + 5, pat=" ", rep="%20"),
        # one entity unescaped in a large text: matches are rare
        dict(name="text_entity", path="device", data="text", n=256 * MiB + 77, pat="&tok0;", rep="&"),
        # deleting a start code from binary data: hardly any match
        dict(name="binary_delete", path="device", data="random", n=1 * GiB, pat="\x00\x00\x01", rep=""),
        # runs of one byte, halved and tripled: every byte is part of a match, with the pattern
        # overlapping itself in the first
        dict(name="run_pairs", path="device", data="run", n=1 * GiB, plen=2, rlen=1),
        dict(name="run_expand", path="device", data="run", n=512 * MiB, plen=1, rlen=3),
        # rule lines of a log dropped to a tag: a long pattern that overlaps itself
        dict(name="rule_lines", path="device", data="rules", n=32 * MiB + 3, plen=40, rlen=4),
        # one call on a document in host memory
        dict(name="unified_doc", path="unified", data="text", n=1 * MiB + 1, pat="&tok0;", rep="&"),
        # a corpus shard through 128 entity pairs, host to host
        dict(name="chain_128", path="chain", data="text", n=64 * MiB + 9, pairs=128),
        # a file larger than one chunk through 8 mixed pairs
        dict(name="stream_8", path="stream", data="text", n=256 * MiB, pairs=8, chunk=32 * MiB),
        # 48 documents with their own pairs in one call
        dict(name="jobs_48", path="jobs", count=48, lo=4 * KiB, hi=4 * MiB),
    ]


def _log_size(rng, lo: int, hi: int) -> int:
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng) -> dict:
    path = rng.choice(["device"] * 9 + ["unified", "chain", "stream", "jobs"])
    if path == "jobs":
        lo = _log_size(rng, 2 * KiB, 64 * KiB)
        return dict(path=path, count=rng.randint(8, 48), lo=lo, hi=lo * rng.randint(8, 64))
    if path == "chain":
        return dict(path=path, data="text", n=_log_size(rng, 64 * KiB, 64 * MiB), pairs=rng.randint(8, 128))
    if path == "stream":
        n = _log_size(rng, 16 * MiB, 256 * MiB)
        return dict(path=path, data="text", n=n, pairs=rng.randint(2, 8), chunk=rng.choice([8, 16, 32, 64]) * MiB)
    data = "text" if path == "unified" else rng.choice(["text", "text", "acgt", "random", "run", "rules"])
    hi = 16 * MiB if path == "unified" else {"rules": 32 * MiB, "text": 256 * MiB}.get(data, 512 * MiB)
    c = dict(path=path, data=data, n=_log_size(rng, 8 * KiB, hi))
    if data == "text":
        c["pat"] = rng.choice([" ", "\n", "e", "&tok%d;" % rng.randrange(128), "word%d" % rng.randrange(200)])
        c["rep"] = "".join(rng.choice("<>%&;_0123456789") for _ in range(rng.randint(0, 6)))
    elif data == "acgt":
        c["pat"] = "".join(rng.choice("ACGT") for _ in range(rng.randint(2, 12)))
        c["rep"] = rng.choice(["", "N", "NNNN", "N" * len(c["pat"])])
    elif data == "random":
        c["pat"] = "".join(chr(rng.randrange(256)) for _ in range(rng.randint(1, 4)))
        c["rep"] = "".join(chr(rng.randrange(256)) for _ in range(rng.randint(0, 4)))
    elif data == "run":
        c["plen"], c["rlen"] = rng.randint(1, 8), rng.randint(0, 8)
        c["rlen"] = min(c["rlen"], 3 * c["plen"])
    else:
        c["plen"], c["rlen"] = rng.randint(33, 64), rng.randint(0, 8)
    return c


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=1)
def _vocabulary():
    """50,000 lowercase words of 1-12 bytes; the same on every machine."""
    rng = np.random.default_rng(3)
    lens = rng.integers(1, 13, size=50_000)
    letters = rng.integers(ord("a"), ord("z") + 1, size=int(lens.sum()), dtype=np.uint8).tobytes()
    ends = np.cumsum(lens)
    return [letters[e - k:e] for e, k in zip(ends.tolist(), lens.tolist())]


def _words(text: str) -> bytes:
    """A literal pattern, or "&tokN;" / "wordN" for the N-th entity token or vocabulary word."""
    if text.startswith("&tok"):
        return W.entity_tokens(3)[int(text[4:-1])]
    if text.startswith("word"):
        return _vocabulary()[int(text[4:])] + b" "
    return text.encode("latin-1")


def _pattern(case: dict, seed: int):
    if case["data"] == "run":
        b = 97 + seed % 26
        return bytes([b]) * case["plen"], bytes(65 + (seed + k) % 26 for k in range(case["rlen"]))
    if case["data"] == "rules":
        return b"-" * case["plen"], b"<hr>...."[:case["rlen"]]
    return _words(case["pat"]), case["rep"].encode("latin-1")


def _pairs(case: dict):
    return W.c3_pairs(3)[:case["pairs"]] if case["path"] == "chain" else W.c4_pairs(4)[:case["pairs"]]


@functools.lru_cache(maxsize=8)
def _tables(special: tuple, device: str):
    words = _vocabulary() + list(special)
    flat = torch.frombuffer(bytearray(b"".join(words)), dtype=torch.uint8).to(device)
    wlen = torch.tensor([len(w) for w in words], dtype=torch.int64, device=device)
    probs = torch.arange(1, 50_001, dtype=torch.float64, device=device) ** -1.1
    probs /= probs.sum()
    mean = float((probs * wlen[:50_000]).sum()) + 1.0
    return flat, wlen, torch.cumsum(wlen, 0) - wlen, torch.cumsum(probs, 0), mean


def _text(n: int, seed: int, device: str, special: tuple, every: int) -> torch.Tensor:
    """Zipf(1.1) words, blanks between them, a line end about every 80 bytes and one of the special
    tokens about every `every` bytes."""
    flat, wlen, wstart, cdf, mean = _tables(special, device)
    g = torch.Generator(device).manual_seed(seed)
    out = torch.empty(n + 32, dtype=torch.uint8, device=device)
    filled = 0
    while filled < n:
        m = int(min(n - filled, 32 * MiB) / mean) + 64
        ids = torch.searchsorted(cdf, torch.rand(m, generator=g, dtype=torch.float64, device=device))
        ids = torch.clamp(ids, max=49_999)
        tok = torch.randint(0, len(special), (m,), generator=g, device=device) + 50_000
        ids = torch.where(torch.rand(m, generator=g, device=device) < mean / every, tok, ids)
        lens = wlen[ids] + 1
        ends = torch.cumsum(lens, 0)
        total = int(ends[-1])
        which = torch.repeat_interleave(torch.arange(m, device=device), lens, output_size=total)
        within = torch.arange(total, device=device) - (ends - lens)[which]
        line = torch.diff(ends // 80, prepend=ends.new_zeros(1)) > 0
        sep = torch.where(line, 10, 32).to(torch.uint8)
        word = ids[which]
        last = within == wlen[word]
        block = torch.where(last, sep[which], flat[torch.where(last, 0, wstart[word] + within)])
        take = min(total, n - filled)
        out[filled:filled + take] = block[:take]
        filled += take
    return out[:n]


def _data(case: dict, n: int, seed: int, device: str) -> torch.Tensor:
    """n bytes on the device, in an allocation that reads up to the next multiple of 16."""
    kind = case["data"]
    if kind == "text":
        return _text(n, seed, device, tuple(W.entity_tokens(3)), 200)
    if kind == "rules":
        k = case["plen"]
        return _text(n, seed, device, (b"-" * k, b"-" * (2 * k), b"=" * k, b"-" * (k // 2)), 400)
    if kind == "run":
        return torch.full((n + 32,), 97 + seed % 26, dtype=torch.uint8, device=device)[:n]
    g = torch.Generator(device).manual_seed(seed)
    if kind == "random":
        return torch.randint(0, 256, (n + 32,), generator=g, dtype=torch.uint8, device=device)[:n]
    letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device=device)
    out = torch.empty(n + 32, dtype=torch.uint8, device=device)
    for a in range(0, n, 64 * MiB):
        m = min(64 * MiB, n - a)
        out[a:a + m] = letters[torch.randint(0, 4, (m,), generator=g, dtype=torch.uint8, device=device).int()]
    return out[:n]


def _jobs(case: dict, seed: int):
    """Documents over their own small alphabets, up to 8 byte strings of each masked by others of the
    same length. Sizes and lengths are the case's, contents the seed's."""
    shape, rng = np.random.default_rng([case["count"], case["lo"], case["hi"]]), np.random.default_rng(seed)
    jobs = []
    for _ in range(case["count"]):
        size = int(math.exp(shape.uniform(math.log(case["lo"]), math.log(case["hi"]))))
        k = int(shape.integers(4, 65))
        alphabet = rng.choice(256, size=k, replace=False).astype(np.uint8)
        data = alphabet[rng.integers(0, k, size=size)].tobytes()
        pairs = []
        for plen in shape.integers(1, 33, size=int(shape.integers(1, 9))).tolist():
            s = int(rng.integers(0, size - plen))
            pairs.append((data[s:s + plen], rng.integers(0, 256, size=plen, dtype=np.uint8).tobytes()))
        jobs.append((data, pairs))
    return jobs


def _host_source(case: dict, lib: CudaReplaceLib, data: torch.Tensor, pairs) -> bytes:
    """The input as host bytes, ended by zero bytes (which no pair matches or writes) up to a fixed
    length of the result, so that results of different seeds can be laid side by side."""
    src = data.cpu().numpy().tobytes()
    if case["path"] == "unified":
        pat, rep = pairs[0]
        length = len(src) + src.count(pat) * (len(rep) - len(pat))
    else:
        with Session(lib, src) as s:
            length = s.apply_batch(pairs)
    return src + bytes(max(0, _result_length(case) - length))


@functools.lru_cache(maxsize=64)
def _ratio(data: str, pairs: tuple) -> float:
    """Output bytes per input byte, from 1 MiB of the same data."""
    out = sample = _data(dict(data=data, plen=len(pairs[0][0])), 1 * MiB, 1, "cpu").numpy().tobytes()
    for p, r in pairs:
        out = out.replace(p, r)
    return len(out) / len(sample)


def _result_length(case: dict) -> int:
    pairs = _pairs(case) if case["path"] in ("chain", "stream") else [_pattern(case, 1)]
    return int(case["n"] * _ratio(case["data"], tuple(pairs)) * 1.01) + 4096


# ------------------------------------------------------------------ one pass
@functools.lru_cache(maxsize=1)
def _lib() -> CudaReplaceLib:
    return CudaReplaceLib()


class _Handle(Session):
    def __del__(self):
        self.close()


def prepare(case: dict, seed: int) -> dict:
    lib = _lib()
    state = dict(path=case["path"], lib=lib)
    if case["path"] == "jobs":
        state["jobs"] = _jobs(case, seed)
        return state
    data = _data(case, case["n"], seed, "cuda")
    if case["path"] in ("chain", "stream"):
        state["pairs"] = _pairs(case)
    else:
        state["pat"], state["rep"] = _pattern(case, seed)
    if case["path"] == "device":
        plen, rlen = len(state["pat"]), len(state["rep"])
        cap = case["n"] + (case["n"] // plen) * max(0, rlen - plen)
        state.update(src=data, out=torch.zeros(cap + 16, dtype=torch.uint8, device="cuda"), cap=cap)
        state["session"] = _Handle(lib, b"")
    else:
        pairs = state.get("pairs") or [(state["pat"], state["rep"])]
        state["src"] = _host_source(case, lib, data, pairs)
        if case["path"] == "chain":
            state["session"] = _Handle(lib, b"")
        elif case["path"] == "stream":
            state["chunk"] = case["chunk"]
    return state


def _array(b: bytes) -> np.ndarray:
    return np.frombuffer(b, dtype=np.uint8) if b else np.empty(0, dtype=np.uint8)


def run(state: dict):
    path, lib = state["path"], state["lib"]
    if path == "device":
        s, src, out = state["session"], state["src"], state["out"]
        s.apply_device_async(src.data_ptr(), src.numel(), state["pat"], state["rep"], out.data_ptr(), state["cap"],
                             torch.cuda.current_stream().cuda_stream)
        return out, s.device_result()  # the buffer; the result's length in it and its matches
    if path == "unified":
        return _array(lib.unified(state["src"], state["pat"], state["rep"]))
    if path == "chain":
        s = state["session"]
        s.reset(state["src"])
        s.apply_batch(state["pairs"])
        return _array(s.result())
    if path == "stream":
        return _array(gpu_replace_streaming(lib, state["src"], state["pairs"], state["chunk"]))
    return [_array(b) for b in replace_jobs(lib, state["jobs"])]


# ------------------------------------------------------------------ what a pass cannot do without
def work(case: dict) -> dict:
    """Input bytes once and output bytes once; the output's share of the input from a sample."""
    if case["path"] == "jobs":
        return {"bytes": 2 * sum(len(d) for d, _ in _jobs(case, 1)), "flops": 0}
    pairs = _pairs(case) if case["path"] in ("chain", "stream") else [_pattern(case, 1)]
    return {"bytes": case["n"] * (1.0 + _ratio(case["data"], tuple(pairs))), "flops": 0}


def exact(case: dict, seed: int):
    """Outputs are bytes and counts, compared as they are: there is no rounded value."""
    return None
