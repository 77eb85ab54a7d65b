"""Declarations, labels and braces around what the straight decoding path takes and what it leaves to the general decoder: every
line alone in a small module, and all of them many times over (as classes); trees and errors against the oracle."""
import pytest

import cases

TYPES = ["u8", "u16", "u32", "u64", "s8", "s16", "s32", "s64", "b8", "b16", "b32", "b64", "b128", "f16", "f16x2", "f32", "f64", "bf16", "pred", "v2 .f32"]
INSIDE = [".%s .%s %%r%s;" % (space, t, tail) for space in ("reg", "local", "param", "shared") for t in TYPES for tail in ("", "<5>")]
INSIDE += [".reg .u32 %%a%s;" % tail for tail in (", %b", ", %b<3>", "<0>", "<4294967295>", "<4294967296>", "<0x10>", "<7U>", "<-1>", "<>", "<5", ",", ", 5", " = 3", "[4]",
                                                  "".join(", %%c%d" % i for i in range(30)))]
INSIDE += [".reg %a;", ".reg .u32 ;", ".reg .u32 add;", ".reg .u32 %envreg3;", ".reg .align 8 .b32 %a;", "L1:", "add:", "%envreg3:", "{ }", "{ { ret; } }", "{ L2: ret; }",
           ".global .u32 x = 3;", ".const .f64 x = 1.5;", ".shared .u32 x = 3;", ".param .b8 p[16];", ".local .align 4 .b8 q[8];"]
OUTSIDE = ["%s.%s .%s x%s;" % (link, space, t, tail) for link in ("", ".visible ", ".extern .weak ") for space in ("global", "const", "shared", "reg") for t in ("u32", "b8", "f64", "pred")
           for tail in ("", " = 7", " = -7", " = 0f3F800000", " = 0d3FF0000000000000", " = 1.25", " = 18446744073709551615", " = 18446744073709551616", " = y", " = WARP_SZ", ", z", "<3>",
                        "[2]", "[2] = {1, 2}", " =", " = 1 2")]


@pytest.mark.parametrize("backend", ["emulation", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_plain_declarations(backend, oracle):
    inside = [cases.HEADER + ".visible .entry k()\n{\n%s\n\tret;\n}\n" % line for line in INSIDE]
    outside = [cases.HEADER + "%s\n.visible .entry k()\n{\n\tret;\n}\n" % line for line in OUTSIDE]
    many = cases.HEADER + "".join(l + "\n" for l in OUTSIDE * 2) + ".visible .entry k()\n{\n" + "".join("%s\n" % l for l in INSIDE * 30) + "\tret;\n}\n"
    texts = inside + outside + [many]
    if backend == "gpu":
        import zluda_b200
        ctx = zluda_b200.Context(0)
        batch = ctx.parse_batch(texts, 1)
        got = [batch.dump(i) for i in range(len(texts))]
        for t in texts[::17] + [many]:      # as a batch of its own: decoded without classes if it is small
            got.append(ctx.parse_batch([t], 1).dump(0))
    else:
        import emu_lib
        got = emu_lib.load().parse(texts, 1)[0]
        got += emu_lib.load().parse(texts[::17] + [many], 1)[0]
    for t, g in zip(texts + texts[::17] + [many], got):
        assert oracle.parse(t, 1)[1] == g, t[-300:]
