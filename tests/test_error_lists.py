"""Error lists that come out of the first decode pass: few and many errors, more than there is room for in that pass, and calls
(whose units always go to the second pass) beside them; trees, error lists and counts against the oracle."""
import pytest

import cases


def module(n_bad, call):
    bad = "\txadd.u32 %r1, %r2, %r3;\n\tadd.u32 %r1, %r2, 7;\n" * n_bad
    callee = ".visible .func f(.param .u32 a)\n{\n\tret;\n}\n" if call else ""
    return cases.HEADER + callee + ".visible .entry k()\n{\n" + bad + ("\tcall.uni f, (%r1);\n\tcall.uni g, (%r1);\n" if call else "") + "\tret;\n}\n"


@pytest.mark.parametrize("backend", ["emulation", pytest.param("gpu", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("n_bad", [0, 1, 63, 2000, 131071, 131072, 140000])
@pytest.mark.parametrize("call", [False, True])
def test_error_lists(backend, n_bad, call, oracle):
    text = module(n_bad, call)
    modes = (0, 1, 2) if n_bad < 100000 else (0,)
    texts = [text, module(3, False), text] if n_bad < 100000 else [text]
    if backend == "gpu":
        import zluda_b200
        ctx = zluda_b200.Context(0)
    else:
        import emu_lib
        emu = emu_lib.load()
    for mode in modes:
        wanted = [oracle.parse(t, mode)[1] for t in texts]
        if backend == "gpu":
            batch = ctx.parse_batch(texts, mode)
            got = [batch.dump(i) for i in range(len(texts))]
            counts = [batch.error_count(i) for i in range(len(texts))]
            assert counts == [int([l for l in d.split("\n") if l.startswith("errors: ")][-1].split()[1]) for d in got]
        else:
            got = emu.parse(texts, mode)[0]
        for a, b in zip(wanted, got):
            assert a == b
