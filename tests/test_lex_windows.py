"""Comments and strings at every place around the lexer's 32-byte windows, 128-byte chunks and 8 KiB tiles: token tables and
lexer errors against the oracle, on the emulation backend and on the GPU."""
import pytest

PIECES = ["// c 12 .5 x::y\n", "/* a/b *** 0x1F \" */", "/*/ not closed yet */", '"s /* // "', "/", "*", "/ /", "12/*x*/U", "%/**/r1", ".5//\n", '""', "a\"b\"c",
          "//", "/*", '"open']      # the last three only end a text


def texts():
    for edge in (32, 128, 8192):
        for piece in PIECES:
            for back in range(0, 7):
                head = ("mov.u32 %r1, 0x2;\n" * (edge // 18 + 1))[:edge - back]
                tail = "" if piece in PIECES[-3:] else "add.f32 %f1, 0f3F800000, .25;\n" * 6
                yield head + piece + tail


@pytest.mark.parametrize("backend", ["emulation", pytest.param("gpu", marks=pytest.mark.gpu)])
def test_comments_and_strings_at_window_edges(backend, oracle):
    if backend == "gpu":
        import zluda_b200
        lexer = zluda_b200.Context(0)
    else:
        import emu_lib
        lexer = emu_lib.load()
    for text in texts():
        assert oracle.lex(text) == lexer.lex(text), text[-80:]
