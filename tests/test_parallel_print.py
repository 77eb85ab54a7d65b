"""Printing a module's bodies in parts: nested blocks, many bodies and one, around the sizes at which a part more is made."""
import pytest

import cases


def module(n_functions, n_words, nested):
    # an add of three registers is seven record words, a block two
    one = "\tadd.u32 %r1, %r2, %r3;\n"
    n = n_words // n_functions // 7
    body = one * n
    if nested:
        depth = 40
        body = ("\t{\n" + one * (n // depth)) * depth + "\t}\n" * depth + one * 5
    head = ".visible .entry k%d(.param .u64 a)\n.maxntid 32, 1, 1\n{\n"
    return cases.HEADER + "".join(head % i + body + "\tret;\n}\n.global .u32 g%d;\n" % i for i in range(n_functions)) + ".visible .func f();\n"


@pytest.mark.gpu
@pytest.mark.parametrize("n_words", [8000, 16200, 16384, 16600, 24700, 66000, 500000])
@pytest.mark.parametrize("n_functions", [1, 7, 200])
@pytest.mark.parametrize("nested", [False, True])
def test_parts(n_words, n_functions, nested, oracle):
    import zluda_b200
    ctx = zluda_b200.Context(0)
    text = module(n_functions, n_words, nested)
    for mode in (0, 1):
        assert ctx.parse_batch([text], mode).dump(0) == oracle.parse(text, mode)[1]
