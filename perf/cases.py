"""The calls that a user of the tokenizer makes, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` gives the fixed ones, ``draw(rng)`` one more of the same ranges,
``prepare`` what a program holds before the call (its text, its tokenizer, its output buffers), ``run`` is one call
through the public entry points, ``work`` the bytes it cannot do without, ``tolerance`` how far another correct
implementation may be off (not at all: token ids, offsets and text are whole numbers).

``call`` says which entry point a case goes through:

  lists      gputok_gpu.GpuTokenizer.tokenize_batch, Python strings in, lists of ids out
  packed     gputok_gpu.GpuTokenizer.encode_packed, Python strings in, arrays out
  host       gputok_b200.Tokenizer.encode, host bytes in, arrays out
  pinned     the same from page-locked memory, the result read in place (a corpus fed through buffer by buffer)
  resident   gputok_b200.Tokenizer.encode_device, text and ids stay in device memory
  noalloc    gputok_b200.Tokenizer.encode_chunks_noalloc, the same without allocations
  decode     gputok_b200.Tokenizer.decode, ids in, bytes out

``text`` says what is tokenised: ``words`` (the generator's English-like ASCII), ``mixed`` (the generator's multi-byte
UTF-8 words and repeated-byte runs) or ``novel`` (lines of a real novel in random order).
"""
from __future__ import annotations

import functools
import gzip
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")
MERGES = os.path.join(GOLDEN, "gpt2_merges.txt")
for _p in (ROOT, os.path.join(ROOT, "gpu-tokenizer_b200")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import gputok_b200  # noqa: E402
from gputok_b200.capi import PinnedArray  # noqa: E402

KiB, MiB = 1 << 10, 1 << 20
MODES = {"opt": gputok_b200.GTK_MODE_OPT, "base": gputok_b200.GTK_MODE_BASE, "localmin": gputok_b200.GTK_MODE_LOCALMIN}
IDS_PER_BYTE = {"words": 0.33, "novel": 0.24, "mixed": 0.6}  # of the GPT-2 table, for work()


def _case(call, nbytes, chunk, text, texts=1, spread="one", mode="opt", gpt2=False):
    """``spread``: how the bytes are cut into texts -- ``one`` text, ``even`` (lengths within a factor of two of
    each other and all different) or ``lognormal`` (median 2 KiB, 64 bytes to 64 KiB)."""
    return {"call": call, "nbytes": int(nbytes), "chunk": int(chunk), "text": text, "texts": int(texts),
            "spread": spread, "mode": mode, "gpt2": bool(gpt2)}


def listed():
    return [
        # one 512-byte string per call, batch size 1: an interactive request, where latency is all that counts
        dict(_case("lists", 512, 2048, "words"), name="one string"),
        # sixteen prompts of about a thousand tokens in one call, lists of ids back: a bucket of the reference's
        # own latency benchmark, and a small serving batch
        dict(_case("lists", 72001, 2048, "novel", 16, "even"), name="sixteen prompts"),
        # ten thousand short records (queries, titles, chat turns) in one call, arrays back
        dict(_case("packed", 5119999, 2048, "words", 10000, "even"), name="ten thousand strings"),
        # one file of a megabyte in 1 KiB chunks from ordinary host memory
        dict(_case("host", MiB, 1024, "words"), name="document"),
        # a corpus that streams through page-locked buffers: what a tokenisation job does all day
        dict(_case("pinned", 96 * MiB + 4711, 4096, "novel"), name="corpus from the host"),
        # text that is in device memory already, in 4 KiB chunks: the throughput benchmark of this repository
        dict(_case("resident", 256 * MiB, 4096, "words"), name="corpus on the device"),
        # long chunks, a fifth of the words outside ASCII, runs of one character: logs, tables, other languages
        dict(_case("resident", 32 * MiB, 32768, "mixed"), name="unicode and runs"),
        # a training shard: documents of very different lengths in one batch, ids for a GPT-2 model
        dict(_case("resident", 64 * MiB - 333, 65536, "mixed", 1, "lognormal", gpt2=True), name="shard of documents"),
        # the sample novel in 2048-byte chunks through the one-block-per-chunk mode: the reference's published run
        dict(_case("host", 711349, 2048, "novel", mode="base"), name="novel, base mode"),
        # the same through the reference's other merge rule, for programs that need the ids it used to give
        dict(_case("host", 711349, 2048, "novel", mode="localmin"), name="novel, local minimum"),
        # chunks on the device inside a serving loop that must not allocate
        dict(_case("noalloc", 2 * MiB, 4096, "novel"), name="no allocation"),
        # ids of a long answer or a checked corpus back to text
        dict(_case("decode", MiB, 2048, "novel"), name="decode"),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("string", "prompts", "strings", "document", "document", "pinned", "resident", "resident",
                       "resident", "base", "localmin", "noalloc", "decode"))
    text = rng.choice(("words", "novel"))
    any_text = rng.choice(("words", "novel", "mixed"))
    short = rng.choice((512, 1024, 2048, 4096, 1000, 3001))
    chunk = rng.choice((short, short, short, 8192))
    if kind == "string":
        return _case("lists", _log(rng, 16, 8 * KiB), 2048, text)
    if kind == "prompts":
        texts = rng.randint(2, 16)
        return _case("lists", texts * _log(rng, 512, 8 * KiB), 2048, text, texts, "even")
    if kind == "strings":
        texts = _log(rng, 100, 20000)
        return _case("packed", texts * _log(rng, 64, 1024), 2048, text, texts, "even")
    if kind == "document":
        return _case("host", _log(rng, 8 * KiB, 7 * MiB), chunk, any_text)
    if kind == "pinned":
        return _case("pinned", _log(rng, 8 * MiB, 128 * MiB), chunk, any_text)
    if kind == "resident":
        spread = rng.choice(("one", "lognormal"))
        chunk = 65536 if spread == "lognormal" else rng.choice((1024, 2048, 4096, 32768))
        return _case("resident", _log(rng, 256 * KiB, 192 * MiB), chunk, any_text, 1, spread, gpt2=rng.random() < 0.3)
    if kind == "base":
        return _case("host", _log(rng, 32 * KiB, 2 * MiB), short, text, mode="base")
    if kind == "localmin":
        return _case("host", _log(rng, 32 * KiB, 2 * MiB), chunk, text, mode="localmin")
    if kind == "noalloc":
        return _case("noalloc", _log(rng, 64 * KiB, 2 * MiB), short, any_text)
    return _case("decode", _log(rng, 1 * KiB, 4 * MiB), 2048, any_text)


@functools.lru_cache(maxsize=None)
def _tokenizer(chunk, gpt2):
    """A program makes its tokenizer once."""
    tok = gputok_b200.Tokenizer(MERGES, chunk_tokens=chunk, device=torch.cuda.current_device())
    tok.set_id_space(gpt2)
    return tok


@functools.lru_cache(maxsize=None)
def _drop_in(chunk):
    import gputok_gpu

    return gputok_gpu.GpuTokenizer(MERGES, chunk)


@functools.lru_cache(maxsize=None)
def _novel_lines():
    with gzip.open(os.path.join(GOLDEN, "pride_and_prejudice.txt.gz")) as f:
        return f.read().splitlines(keepends=True)


def _text(kind, nbytes, seed):
    """uint8 array of that many bytes."""
    if kind != "novel":
        mix = gputok_b200.MIX_STRESS if kind == "mixed" else gputok_b200.MIX_PLAIN
        return gputok_b200.TextGen(seed).text(nbytes, mix=mix)
    lines = _novel_lines()
    rng, parts, have = np.random.default_rng(seed), [], 0
    while have < nbytes:  # the whole novel, its lines in another order each time
        one = b"".join([lines[i] for i in rng.permutation(len(lines))])
        parts.append(one[: nbytes - have])
        have += len(parts[-1])
    return np.frombuffer(b"".join(parts), dtype=np.uint8)


def _offsets(case, seed):
    """int64[T+1]: where the texts start and end."""
    n = case["nbytes"]
    if case["spread"] == "lognormal":
        return gputok_b200.TextGen.lognormal_offsets(seed, n)
    if case["spread"] == "one":
        return np.array([0, n], dtype=np.int64)
    cuts = np.random.default_rng(seed).uniform(0.7, 1.4, case["texts"]).cumsum()
    return np.concatenate([[0], np.round(cuts * (n / cuts[-1]))]).astype(np.int64)


BASE_SEED = 11


def _shuffled_chunks(case, seed):
    """One text whose whole chunks stand in another order for every seed.  Chunks are tokenised each for itself, so
    the number of ids, which is the length of the arrays that the call returns, stays the same."""
    chunk, n = case["chunk"], case["nbytes"]
    data = np.array(_text(case["text"], n, BASE_SEED))
    whole = data[: n - n % chunk].reshape(-1, chunk)
    whole[:] = whole[np.random.default_rng(seed).permutation(len(whole))]
    return data


def prepare(case, seed):
    call, n, chunk = case["call"], case["nbytes"], case["chunk"]
    state = {"call": call, "mode": MODES[case["mode"]]}
    if call in ("lists", "packed"):
        # arrays are returned whole: the same strings in another order, for the reason given above
        of = BASE_SEED if call == "packed" else seed
        data, off = _text(case["text"], n, of), _offsets(case, of)
        texts = [data[a:b].tobytes().decode("utf-8", "ignore") for a, b in zip(off[:-1], off[1:])]
        state["tok"] = _drop_in(chunk)
        if call == "packed":
            state["texts"] = [texts[i] for i in np.random.default_rng(seed).permutation(len(texts))]
            return state
        state["texts"] = texts
        # what a model is fed with: one padded row for each prompt, as wide as an id for every byte could ask for
        state["padded"] = np.zeros((len(texts), 2 * n // len(texts) + 16), dtype=np.int32)
        state["lengths"] = np.zeros(len(texts), dtype=np.int64)
        return state
    state["tok"] = tok = _tokenizer(chunk, case["gpt2"])
    if call == "host":
        state["data"], state["off"] = _shuffled_chunks(case, seed), _offsets(case, seed)
        return state
    if call == "pinned":
        state["pin"], state["off"] = PinnedArray(n), _offsets(case, seed)
        state["pin"].array[:] = _shuffled_chunks(case, seed)
        return state
    data, off = _text(case["text"], n, seed), _offsets(case, seed)
    if call == "decode":
        state["ids"] = tok.encode(data, off)[0]
        return state
    chunk_cap = n // chunk + len(off) + 1
    if call == "noalloc":
        off = np.minimum(np.arange(0, n + chunk, chunk, dtype=np.int64), n)
        state["counts"] = torch.zeros(len(off) - 1, dtype=torch.int32, device="cuda")
    elif case["spread"] == "lognormal":
        chunk_cap = n // chunk + n // 64 + 2  # no text is shorter than 64 bytes
    state["n"], state["chunk"], state["n_off"] = n, chunk, len(off) - 1
    state["bytes"] = torch.from_numpy(data.copy()).cuda()
    state["off"] = torch.from_numpy(off).cuda()
    state["ids"] = torch.zeros(n, dtype=torch.int32, device="cuda")  # an id for every byte at the most
    state["chunk_off"] = torch.zeros(chunk_cap, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()  # the tokenizer works on a stream of its own
    return state


def run(state):
    call, tok = state["call"], state["tok"]
    if call == "lists":
        batch, _ = tok.tokenize_batch(state["texts"])
        padded, lengths = state["padded"], state["lengths"]
        for i, ids in enumerate(batch):
            padded[i, : len(ids)] = ids
            lengths[i] = len(ids)
        return padded, lengths
    if call == "packed":
        ids, text_off, chunk_off, _ = tok.encode_packed(state["texts"])
        return ids, text_off, chunk_off
    if call == "host":
        return tok.encode(state["data"], state["off"], mode=state["mode"])[:3]
    if call == "pinned":
        return tok.encode(state["pin"].array, state["off"], mode=state["mode"], copy=False)[:3]
    if call == "decode":
        return np.frombuffer(tok.decode(state["ids"]), dtype=np.uint8)
    ids, chunk_off = state["ids"], state["chunk_off"]
    if call == "noalloc":
        tok.encode_chunks_noalloc(state["bytes"].data_ptr(), state["n"], state["off"].data_ptr(), state["n_off"],
                                  state["chunk"], ids.data_ptr(), state["counts"].data_ptr())
        return ids, state["counts"]
    n_ids, n_chunks, _ = tok.encode_device(state["bytes"].data_ptr(), state["n"], state["off"].data_ptr(),
                                           state["n_off"], ids.data_ptr(), len(ids), chunk_off.data_ptr(),
                                           len(chunk_off), mode=state["mode"])
    return ids, chunk_off, n_ids, n_chunks


def work(case):
    """Text once, ids once (int32, as many as the text has by experience) and, except for decoding, one int64 offset
    in per text and one out per chunk."""
    n = case["nbytes"]
    texts = max(case["texts"], n // 3300 if case["spread"] == "lognormal" else 1)
    offsets = 0 if case["call"] == "decode" else 8 * (2 * texts + n // case["chunk"] + 2)
    return {"bytes": n + 4 * IDS_PER_BYTE[case["text"]] * n + offsets, "flops": 0}


def tolerance(case):
    return "exact"
