"""What users of the PTX front end ask of it, as cases that can be timed.

A case goes through the package's public entry points, host text in and host records out unless the entry point itself
works on device memory:

  single    parse_module_checked / parse_module_unchecked / parse_for_errors on one module (a JIT compiling one kernel)
  batch     Context.parse_batch and the verdict of every module (a fatbin extractor, a precompiler, a service), with the
            records left where the library puts them and, for the modules with errors, their error lists
  resident  Context.run + Context.fetch on text that was staged before (a caller that keeps its text on the device)
  lexer     ptxfe_lex_device_noalloc on device memory (a caller that may not allocate)

Text is synthetic (zluda_b200.corpus); sizes are those of the repository's own configurations and everything below them.
So that the records of a case have the same number whatever the seed, batches of kernels and debug modules keep their
statements and take their values from the seed: the order of the modules, and the digits A to F of hexadecimal literals.
"""
import ctypes
import random
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import zluda_b200
from zluda_b200 import corpus

MODES = {"checked": zluda_b200.CHECKED, "unchecked": zluda_b200.UNCHECKED, "errors": zluda_b200.ERRORS_ONLY}

# Record bytes and dump bytes per byte of text (what comes back for what is read)
RECORDS = {"kernels": 1.06, "literals": 1.43, "debug": 0.61}
DUMP = 4.9
# Tokens per byte of text
TOKENS = 0.28


def _case(kind, text, n_bytes, modules=1, mode="checked", memory="pageable", damaged=0.0):
    """kind as above; text: kernels (instruction streams), literals (data tables) or debug (-lineinfo, scopes, comments);
    n_bytes of text over all modules (roughly: the generators work in statements); memory: pinned (one page-locked
    buffer, modules back to back) or pageable (one bytes object per module); damaged: share of modules with errors."""
    return {"kind": kind, "text": text, "bytes": int(n_bytes), "modules": int(modules), "mode": mode, "memory": memory, "damaged": damaged}


def listed():
    rows = [
        # the smallest call: a JIT hands over one small kernel, latency is everything
        ("one_small_kernel", _case("single", "kernels", 2000)),
        # one module of the batch configuration's median size
        ("one_module", _case("single", "kernels", 131 * 1000)),
        # the error list of one module with a few bad statements (an editor, a test suite)
        ("errors_of_one_module", _case("single", "kernels", 40 * 1000, mode="errors", damaged=1.0)),
        # one program of many kernels: 64 entries, ~4.6 MB
        ("one_program", _case("batch", "kernels", 4600 * 1000, memory="pinned")),
        # a library's worth of small kernels, each a file of its own
        ("small_files", _case("batch", "kernels", 20 * 1000 * 1000, modules=6000)),
        # a precompiler with --ignore-errors: files from disk, some with statements that the grammar does not know
        ("precompile_ignore_errors", _case("batch", "kernels", 11 * 1000 * 1000, modules=85, mode="unchecked", damaged=0.1)),
        # one fatbin's worth of modules
        ("fatbin", _case("batch", "kernels", 64 << 20, modules=250, memory="pinned")),
        # the benchmark configuration: 4,096 modules, 1 GiB
        ("fatbin_scale", _case("batch", "kernels", 1 << 30, modules=4096, memory="pinned")),
        # constant tables: huge initialiser lists, hex and decimal, and float constants
        ("literal_tables", _case("batch", "literals", 39 * 1000 * 1000, memory="pinned")),
        # -lineinfo output: .loc before every instruction, comments, nested scopes, calls
        ("debug_info", _case("batch", "debug", 33 * 1000 * 1000, memory="pinned")),
        # text kept on the device, parsed there, records fetched
        ("resident", _case("resident", "kernels", 130 * 1000 * 1000, modules=500, memory="pinned")),
        # the lexer for callers that cannot allocate
        ("lexer_no_alloc", _case("lexer", "kernels", 3 * 1000 * 1000)),
    ]
    return [dict(c, name=name) for name, c in rows]


BASE_SEED = 1001


def _new_digits(seed):
    """A translation of bytes that permutes A to F (hexadecimal literals are the only words that hold them)."""
    new = list(b"ABCDEF")
    random.Random(seed).shuffle(new)
    return bytes.maketrans(b"ABCDEF", bytes(new))


def _digits(text, seed):
    return text.translate(_new_digits(seed))


def _digits_in_place(blob, spans, seed):
    table = np.frombuffer(_new_digits(seed), np.uint8)

    def one(part):
        np.take(table, blob[part[0]:part[1]], out=blob[part[0]:part[1]], mode="clip")

    end = spans[-1][0] + spans[-1][1]
    step = 4 << 20
    with ThreadPoolExecutor(16) as pool:
        list(pool.map(one, [(a, min(end, a + step)) for a in range(0, end, step)]))


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    use = rng.choice(("single", "single", "single", "batch", "batch", "batch", "batch", "literals", "debug", "resident", "lexer"))
    if use == "single":
        mode = rng.choice(("checked", "checked", "unchecked", "errors"))
        damaged = 1.0 if mode == "errors" or (mode == "unchecked" and rng.random() < 0.5) else 0.0
        return _case("single", "kernels", _log_uniform(rng, 1100, 600 * 1000), mode=mode, damaged=damaged)
    if use == "literals":
        return _case("batch", "literals", _log_uniform(rng, 12000, 128 << 20), memory=rng.choice(("pinned", "pageable")))
    if use == "debug":
        return _case("batch", "debug", _log_uniform(rng, 100 * 1000, 128 << 20), memory=rng.choice(("pinned", "pageable")))
    if use == "resident":
        modules = _log_uniform(rng, 1, 2000)
        return _case("resident", "kernels", _log_uniform(rng, max(20000, 2000 * modules), 256 << 20), modules=modules, memory="pinned")
    if use == "lexer":
        return _case("lexer", "kernels", _log_uniform(rng, 2000, 15 << 20))
    # batches: modules of at least 2 KB and at most 8 MiB each, pinned ones up to 1 GiB in all
    memory = rng.choice(("pinned", "pageable"))
    modules = _log_uniform(rng, 1, 10000 if memory == "pinned" else 6000)
    mode = rng.choice(("checked", "checked", "checked", "unchecked"))
    damaged = rng.choice((0.02, 0.1, 0.3)) if mode == "unchecked" and memory == "pageable" and modules <= 600 else 0.0
    top = min((1 << 30) if memory == "pinned" else (128 << 20), modules * (8 << 20))
    if damaged:
        top = max(2000 * modules, int(min(top, 1200 * 1000 / damaged)))
    return _case("batch", "kernels", _log_uniform(rng, max(4000, 2000 * modules), max(4000, top)), modules=modules, mode=mode, memory=memory, damaged=damaged)


def _damage(text, rng):
    """One to four statements of the module spoilt the ways that real files have them: an instruction or a modifier that
    the grammar does not know, an operand that is missing, once in a while a byte that no token starts with."""
    lines = text.split(b"\n")
    body = [i for i, line in enumerate(lines) if line.startswith(b"\t") and line.endswith(b";") and b", " in line and b"." in line and b"{" not in line]
    for i in rng.sample(body, min(len(body), rng.randint(1, 4))):
        line, way = lines[i], rng.random()
        if way < 0.4:
            line = b"\tx" + line[1:]
        elif way < 0.7:
            at = line.index(b".")
            line = line[:at] + b".q8" + line[at:]
        elif way < 0.95:
            line = line[:line.rindex(b", ")] + b";"
        else:
            line = line[:-1] + b"`;"
        lines[i] = line
    return b"\n".join(lines)


def _one_text(case, seed):
    """The single module of a literals or debug case."""
    n = case["bytes"]
    if case["text"] == "literals":
        # 16 arrays (fewer in small modules) and constants in the proportion of the literal-heavy configuration
        arrays = max(1, min(16, n // 40000))
        init = max(64, int(n * 0.88 / (arrays * 8.0)))
        return corpus.config2(seed, arrays, init, max(16, int(n * 0.12 / 44)))[0]
    return _digits(corpus.config3(BASE_SEED, n, max(2, min(64, n // 16000)), max(2, n * 20000 >> 28))[0], seed)


class State:
    """What a user's program holds: its texts in the form that it passes them in, and the context that it keeps."""


_context = None


def _shared_context():
    # a program keeps one context for all its batches
    global _context
    if _context is None:
        _context = zluda_b200.Context(0)
    return _context


def prepare(case, seed):
    s = State()
    s.case, s.mode = case, MODES[case["mode"]]
    rng = random.Random(seed)
    n = case["modules"]
    if case["text"] != "kernels":
        texts = [_one_text(case, seed)]
        total = len(texts[0])
    else:
        bound = corpus.config1_total_bound(seed, n, case["bytes"])
        s.buffer = torch.empty(bound, dtype=torch.uint8, pin_memory=case["memory"] == "pinned")
        blob = s.buffer.numpy()
        own = case["kind"] in ("single", "lexer")
        order = list(range(n))
        rng.shuffle(order)
        spans = corpus.config1_into(blob, seed if own else BASE_SEED, n, case["bytes"], order)
        if not own:
            _digits_in_place(blob, spans, seed)
        if case["memory"] != "pinned":
            texts = [blob[o:o + k].tobytes() for o, k in spans]
            s.buffer = None
    if case["damaged"]:
        where = list(range(n)) if own else [order.index(m) for m in range(n)]
        spoil = rng if own else random.Random(BASE_SEED)
        for m in where:
            if spoil.random() < case["damaged"] or n == 1:
                texts[m] = _damage(texts[m], spoil)
    if case["memory"] == "pinned":
        if case["text"] != "kernels":
            s.buffer = torch.empty(total, dtype=torch.uint8, pin_memory=True)
            s.buffer.numpy()[:] = np.frombuffer(texts[0], np.uint8)
            spans = [(0, total)]
        base = s.buffer.data_ptr()
        s.texts = zluda_b200.Texts([(base + o, k) for o, k in spans])
        s.n = len(spans)
    else:
        s.texts, s.n = texts, len(texts)
    if case["kind"] == "single":
        s.texts = texts[0].decode()
    elif case["kind"] == "batch":
        s.context = _shared_context()
    elif case["kind"] == "resident":
        s.context = zluda_b200.Context(0)
        s.context.stage(s.texts)
    elif case["kind"] == "lexer":
        # room for one token per two bytes, as a caller without a count has to provide
        s.text = torch.frombuffer(bytearray(texts[0]), dtype=torch.uint8).cuda()
        s.tokens = torch.zeros(case["bytes"] // 2 + 1024, dtype=torch.int64, device="cuda")
        s.counts = torch.zeros(2, dtype=torch.int32, device="cuda")
        lex = zluda_b200.lib().ptxfe_lex_device_noalloc
        lex.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_uint64, ctypes.c_void_p, ctypes.c_void_p]
        s.lex = lex
    return s


def _records(batch, n, context):
    """The records of all modules as one array over the library's own result memory (modules follow one another)."""
    at = zluda_b200.lib().ptxfe_module_records
    first, last, count, base = ctypes.POINTER(ctypes.c_uint32)(), ctypes.POINTER(ctypes.c_uint32)(), ctypes.c_uint64(), ctypes.c_uint64()
    at(batch._h, 0, ctypes.byref(first), ctypes.byref(count), ctypes.byref(base))
    at(batch._h, n - 1, ctypes.byref(last), ctypes.byref(count), ctypes.byref(base))
    begin = ctypes.cast(first, ctypes.c_void_p).value
    words = (ctypes.cast(last, ctypes.c_void_p).value - begin) // 4 + count.value
    array = (ctypes.c_int32 * words).from_address(begin)
    array.owner = (batch, context)          # the memory is the context's
    return np.frombuffer(array, np.int32)


def _bytes_of(text, room=0):
    """The text as an array, with zeros behind it where the caller wants the same length whatever the text."""
    b = text.encode()
    if not room:
        return np.frombuffer(b, np.uint8)
    a = np.zeros(max(room, len(b)), np.uint8)
    a[:len(b)] = np.frombuffer(b, np.uint8)
    return a


def run(state):
    kind = state.case["kind"]
    if kind == "single":
        mode = state.case["mode"]
        if mode == "errors":
            return {"errors": _bytes_of("\n".join(zluda_b200.parse_for_errors(state.texts)), 4096)}
        parse = zluda_b200.parse_module_checked if mode == "checked" else zluda_b200.parse_module_unchecked
        r = parse(state.texts)
        return {"ok": r.ok, "dump": _bytes_of(r.dump, 8 * state.case["bytes"]), "errors": _bytes_of("\n".join(r.errors), 4096)}
    if kind == "lexer":
        stream = torch.cuda.current_stream().cuda_stream
        status = state.lex(0, state.text.data_ptr(), state.text.numel(), state.tokens.data_ptr(), state.tokens.numel(), state.counts.data_ptr(), stream)
        return {"status": status, "tokens": state.tokens, "counts": state.counts}
    if kind == "resident":
        state.context.run(state.mode)
        batch = state.context.fetch()
    else:
        batch = state.context.parse_batch(state.texts, state.mode)
    out = {"status": np.array([batch.status(i) for i in range(state.n)], np.int32)}
    if state.case["damaged"]:
        counts = [batch.error_count(i) for i in range(state.n)]
        out["error_counts"] = np.array(counts, np.int32)
        out["errors"] = _bytes_of("\n".join("\n".join(batch.errors(i)) for i in range(state.n) if counts[i]))
    out["records"] = _records(batch, state.n, state.context)
    return out


def work(case):
    n = case["bytes"]
    if case["kind"] == "single":
        return {"bytes": n * (1 if case["mode"] == "errors" else 1 + DUMP), "flops": 0}
    if case["kind"] == "lexer":
        return {"bytes": n * (1 + 8 * TOKENS), "flops": 0}
    return {"bytes": n * (1 + RECORDS[case["text"]]), "flops": 0}


def tolerance(case):
    return "exact"
