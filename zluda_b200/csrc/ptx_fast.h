// The straight path through the decoder, for what most statements are: an instruction whose operands are names, packs of
// names, [name + offset] and literals, a declaration of variables, a label, a brace, or a kernel header whose parameters are
// plain scalars.
//
// The general decoder (ptx_decode.h) keeps its state in an object in memory, backtracks and reports errors; a mov with two
// registers is 2,500 instructions there, most of them waiting for that object (40,000 cycles for a lone warp).  Here the
// state is a few registers, nothing is undone and nothing is reported: the function either produces the very record that
// the general decoder would, or returns 0 and the general decoder starts over.  It gives up on anything out of the
// ordinary - an error, an optional operand that would need backtracking, `call`, `%envreg`, names that are opcodes.
// (The first decode step of a 2 KB kernel: 86 us without it.)
// (Declarations: 100,000 constants 199 -> 138 us, the headers and registers of 6,000 small files 246 -> 153.)
#pragma once
#include "ptx_units.h"

struct PtxFast {
    const uint8_t* text;
    const PtxTokenWord* tokens;      // the unit's first token
    const PtxTokenWord* win;         // the same in fast memory: win_n of them, win_stride apart
    uint32_t win_n, win_stride;
    uint32_t n;                      // tokens of the unit
    // where the record goes: word k to words[k * stride], its tag to tags[k * stride] (nullptr: none)
    uint32_t* words;
    uint32_t* tags;
    uint32_t stride, cap;
    uint32_t nw = 0;
    bool ok = true;
    // of a function header
    uint32_t name_tok = 0, n_inputs = 0;

    PTX_HD PtxTokenWord tk(uint32_t i) const { return i < win_n ? win[i * win_stride] : tokens[i]; }
    PTX_HD uint32_t kind(uint32_t i) const { return i < n ? tk(i).y >> 16 : 0xFFFEu; }
    PTX_HD void w(uint32_t x, uint32_t tag = 0) {
        if (nw < cap) {
            words[nw * stride] = x;
            if (tags) tags[nw * stride] = tag;
        }
        nw++;
    }
    PTX_HD void span(uint32_t i) {
        const PtxTokenWord t = tk(i);
        w(t.x, (PTX_TAG_START << 8) | i);
        w(t.y & 0xFFFFu, (PTX_TAG_LEN << 8) | i);
    }
    PTX_HD void name(uint32_t head, uint32_t i) {
        const PtxTokenWord t = tk(i);
        w(head | ((t.y & 0xFFFFu) << 8), (PTX_TAG_NAMEHEAD << 8) | i);
        w(t.x, (PTX_TAG_START << 8) | i);
    }
    // a plain identifier: no opcode, no %envreg (an error for the general decoder to report), a length that fits
    PTX_HD bool ident(uint32_t i) const {
        if (i >= n) return false;
        const PtxTokenWord t = tk(i);
        const uint32_t len = t.y & 0xFFFFu;
        if ((t.y >> 16) != T_IDENT || len == 0xFFFFu) return false;
        return !((len == 8 || len == 9) && ptx_envreg_number(text + t.x, len));
    }
    PTX_HD static bool numeric(uint32_t k) { return k == T_DECIMAL || k == T_HEX; }

    // ---- operands
    enum { F_NAME = 1, F_OFFSET = 2, F_IMM = 3, F_PACK = 4, F_BAD = 0xFF };
    struct Operand {
        uint8_t form, neg, kind, n;      // kind: of an immediate; n: names in a pack
        uint32_t at, lit;                // first token; the literal
        uint64_t bits;
    };
    // 1 = an operand, 0 = none starts here, -1 = not for this path
    PTX_HD int operand(uint32_t& i, Operand& o) const {
        const uint32_t k = kind(i);
        o.at = i;
        o.neg = 0;
        if (k == T_IDENT) {
            if (!ident(i)) return -1;
            i++;
            const uint32_t k1 = kind(i);
            if (k1 == T_DOTIDENT) return -1;
            o.form = F_NAME;
            if (k1 != T_PLUS) return 1;
            uint32_t j = i + 1;
            if (kind(j) == T_MINUS) { o.neg = 1; j++; }
            if (!numeric(kind(j))) return -1;
            const PtxTokenWord t = tk(j);
            uint64_t mag;
            if ((t.y & 0xFFFFu) == 0xFFFFu || (ptx_literal_scan(text + t.x, t.y & 0xFFFFu, (uint16_t)(t.y >> 16), &mag) & (PTX_LC_ERR | PTX_LC_GT_I32))) return -1;
            o.form = F_OFFSET;
            o.lit = j;
            o.bits = o.neg ? 0 - mag : mag;
            i = j + 1;
            return 1;
        }
        if (k == T_MINUS || numeric(k) || k == T_F32HEX || k == T_F64HEX || k == T_F64) {
            uint32_t j = i;
            if (k == T_MINUS) {
                o.neg = 1;
                if (!numeric(kind(++j))) return -1;
            }
            const PtxTokenWord t = tk(j);
            const uint32_t len = t.y & 0xFFFFu, kd = t.y >> 16;
            if (len == 0xFFFFu) return -1;
            if (kd == T_F64) {
                o.kind = 3;
                o.bits = ptx_parse_f64(text + t.x, len);
            } else {
                uint64_t mag;
                const uint32_t code = ptx_literal_scan(text + t.x, len, (uint16_t)kd, &mag);
                if (code & PTX_LC_ERR || (o.neg && (code & PTX_LC_GT_2P63))) return -1;
                o.kind = kd == T_F32HEX ? 2 : kd == T_F64HEX ? 3 : o.neg ? 1 : code & (PTX_LC_UNS | PTX_LC_GT_I63) ? 0 : 1;
                o.bits = o.neg ? 0 - mag : mag;
            }
            o.form = F_IMM;
            o.lit = j;
            i = j + 1;
            return 1;
        }
        if (k == T_LBRACE) {
            uint32_t j = i + 1, c = 0;
            for (;;) {
                if (c == 8 || !ident(j)) return -1;
                c++;
                const uint32_t k1 = kind(j + 1);
                j += 2;
                if (k1 == T_RBRACE) break;
                if (k1 != T_COMMA) return -1;
            }
            o.form = F_PACK;
            o.n = (uint8_t)c;
            i = j;
            return 1;
        }
        return k == T_WARP_SZ || PtxDecoder::is_opcode((uint16_t)k) ? -1 : 0;
    }
    PTX_HD void put_operand(const Operand& o) {
        switch (o.form) {
        case F_NAME: name(OPK_REG, o.at); break;
        case F_OFFSET:
            name(OPK_REG_OFFSET, o.at);
            w((uint32_t)o.bits, ((o.neg ? PTX_TAG_NEG_LO : PTX_TAG_VAL_LO) << 8) | o.lit);
            break;
        case F_IMM:
            w(OPK_IMM | ((uint32_t)o.kind << 4));
            w((uint32_t)o.bits, ((o.neg ? PTX_TAG_NEG_LO : PTX_TAG_VAL_LO) << 8) | o.lit);
            w((uint32_t)(o.bits >> 32), ((o.neg ? PTX_TAG_NEG_HI : PTX_TAG_VAL_HI) << 8) | o.lit);
            break;
        default:
            w(OPK_VEC_PACK | ((uint32_t)o.n << 4));
            for (uint32_t k = 0; k < o.n; k++) name(0, o.at + 1 + 2 * k);
            break;
        }
    }
    // what the pattern bodies build with: data bytes first, then operands, in the order of the record
    struct Builder {
        uint8_t data[24];
        uint8_t n_data = 0, n_args = 0;
        int8_t args[PTX_MAX_ARGS];
        bool ok = true;
        PTX_HD void put(uint32_t x) {
            if (x >= 0xFFu || n_data == sizeof data || n_args) { ok = false; return; }
            data[n_data++] = (uint8_t)x;
        }
        PTX_HD void arg(int i) {
            if (n_args == PTX_MAX_ARGS) { ok = false; return; }
            args[n_args++] = (int8_t)i;
        }
        PTX_HD void arg_imm_u64(uint64_t) { ok = false; }
        PTX_HD void err(int, int, uint32_t, uint32_t) { ok = false; }
        PTX_HD void err_todo(int) { ok = false; }
        PTX_HD bool op_as_u64(int, uint64_t*) { ok = false; return false; }
        PTX_HD bool op_as_f64(int, double*) { ok = false; return false; }
        PTX_HD void op_span(int, uint32_t*, uint32_t*) { ok = false; }
    };

    // One instruction statement, all of the unit's tokens.  Returns true with the record written (nw words).
    PTX_HD bool instruction() {
        if (n < 2 || n > 250 || kind(n - 1) != T_SEMI) return false;
        uint32_t i = 0, head = 0, pred = 0;
        if (kind(0) == T_AT) {
            i = 1;
            head = 1;
            if (kind(1) == T_EXCL) { head = 3; i = 2; }
            if (!ident(i)) return false;
            pred = i++;
        }
        const uint32_t opk = kind(i);
        if (!PtxDecoder::is_opcode((uint16_t)opk)) return false;
        const uint32_t at_op = i++;
        const PtxOpcode op = ptx_opcodes[opk - T_OP_FIRST];
        w(0);
        if (head) span(pred);
        uint32_t variant;
        if (op.special == 1) {
            if (kind(i) == T_MOD_uni) i++;
            if (kind(i) != T_IDENT || (tk(i).y & 0xFFFFu) == 0xFFFFu || i + 2 != n) return false;
            span(i);
            variant = I_Bra;
        } else {
            if (op.special) return false;
            // a name with a ':' behind it is a label even if it is an opcode
            if (kind(at_op + 1) == T_COLON && at_op == 0) return false;
            const uint32_t mb = i;
            uint64_t m[3] = {0, 0, 0};
            for (; PtxDecoder::is_modifier((uint16_t)kind(i)); i++) {
                const uint32_t x = kind(i) - T_MOD_FIRST;
                const uint64_t bit = 1ull << (x & 63u);
                m[0] |= x < 64 ? bit : 0;
                m[1] |= x >= 64 && x < 128 ? bit : 0;
                m[2] |= x >= 128 ? bit : 0;
            }
            const uint32_t me = i;
            int pattern = -1;
            for (int c = 0; c < op.n_chain && pattern < 0; c++) {
                const PtxChain ch = ptx_chains[op.first_chain + c];
                if (ch.is_default || (m[0] & ch.key[0]) || (m[1] & ch.key[1]) || (m[2] & ch.key[2])) pattern = ch.pattern;
            }
            if (pattern < 0) return false;
            const PtxPattern pt = ptx_patterns[pattern];
            int mv[PTX_MAX_SLOTS];
            const int n_slots = pt.n_unordered + pt.n_ordered;
            for (int s = 0; s < n_slots; s++) mv[s] = (pt.typed_mask >> s) & 1 ? -1 : 0;
            uint32_t end = me, seen = 0;
            for (int s = n_slots - 1; s >= pt.n_unordered; s--) {
                const PtxSlot sl = ptx_slots[pt.first_slot + s];
                const int v = end > mb ? ptx_set_value[sl.set][kind(end - 1) - T_MOD_FIRST] : -1;
                if (v >= 0) { mv[s] = v; end--; }
                else if (!sl.optional) return false;
            }
            for (uint32_t j = mb; j < end; j++) {
                const uint32_t place = ptx_mod_place[pattern][kind(j) - T_MOD_FIRST];
                const uint32_t bit = place ? 1u << ((place >> 8) - 1) : 0u;
                if (!place || (seen & bit)) return false;
                seen |= bit;
                mv[(place >> 8) - 1] = (int)(place & 0xFFu);
            }
            if (pt.required_mask & ~seen) return false;
            // operands; an optional one that is not there is absent, one that would have to be tried both ways is not for here
            Operand ops[PTX_MAX_ARGS];
            int av[PTX_MAX_ARGS], aneg[PTX_MAX_ARGS], auni[PTX_MAX_ARGS];
            int n_ops = 0;
            for (int a = 0; a < pt.n_args; a++) {
                const uint32_t fl = ptx_pattern_args[pt.first_arg + a];
                const uint32_t save = i;
                bool there = true;
                aneg[a] = auni[a] = 0;
                av[a] = -1;
                auto eat = [&](uint32_t k) { if (kind(i) != k) return false; i++; return true; };
                if (!(a == 0 || (fl & PTX_ARG_PRE_PIPE))) there = eat(T_COMMA);
                if (there && (fl & PTX_ARG_PRE_BRACKET)) there = eat(T_LBRACKET);
                if (there && (fl & PTX_ARG_PRE_PIPE)) there = eat(T_PIPE);
                if (there && (fl & PTX_ARG_NEGATED)) aneg[a] = eat(T_EXCL) ? 1 : 0;
                if (there) {
                    const int r = operand(i, ops[n_ops]);
                    if (r < 0) return false;
                    there = r > 0;
                    if (there && (fl & PTX_ARG_POST_BRACKET)) there = eat(T_RBRACKET);
                    if (there && (fl & PTX_ARG_UNIFIED)) auni[a] = eat(T_MOD_unified) ? 1 : 0;
                }
                if (there) { av[a] = n_ops++; continue; }
                if (!(fl & PTX_ARG_OPTIONAL)) return false;
                i = save;
                aneg[a] = auni[a] = 0;
            }
            if (i + 1 != n) return false;
            Builder b;
            ptx_build(pattern, b, mv, av, aneg, auni);
            if (!b.ok) return false;
            for (uint32_t k = 0; k < b.n_data; k += 4) {
                uint32_t x = 0;
                for (uint32_t q = 0; q < 4 && k + q < b.n_data; q++) x |= (uint32_t)b.data[k + q] << (8 * q);
                w(x);
            }
            for (uint32_t k = 0; k < b.n_args; k++) {
                if (b.args[k] < 0) w(PTX_ABSENT);
                else put_operand(ops[b.args[k]]);
            }
            variant = pt.instr;
        }
        if (nw > cap) return false;
        words[0] = (uint32_t)U_INSTR | ((nw - 1) << 8) | (variant << 22) | (head << 29);
        return true;
    }

    PTX_HD static int scalar_of(uint32_t k) {
        switch (k) {
        case T_MOD_u64: return ScalarType_U64;
        case T_MOD_u32: return ScalarType_U32;
        case T_MOD_b64: return ScalarType_B64;
        case T_MOD_b32: return ScalarType_B32;
        case T_MOD_f32: return ScalarType_F32;
        case T_MOD_f64: return ScalarType_F64;
        case T_MOD_s32: return ScalarType_S32;
        case T_MOD_s64: return ScalarType_S64;
        case T_MOD_u16: return ScalarType_U16;
        case T_MOD_u8: return ScalarType_U8;
        case T_MOD_pred: return ScalarType_Pred;
        case T_MOD_b16: return ScalarType_B16;
        case T_MOD_b8: return ScalarType_B8;
        case T_MOD_f16: return ScalarType_F16;
        case T_MOD_s16: return ScalarType_S16;
        case T_MOD_s8: return ScalarType_S8;
        default: return -1;
        }
    }
    // type name, name, ... ;   or   type name<count>;   or (`initial`) type name = literal;   from token i on, of a variable that
    // is no array: the multivariable record
    PTX_HD bool variables(uint32_t i, uint32_t space, bool initial, bool one) {
        const int scalar = scalar_of(kind(i));
        if (scalar < 0) return false;
        const uint32_t at = nw;
        nw += 3;
        uint32_t names = 0, count = 0;
        for (;;) {
            if (!ident(++i)) return false;
            span(i);
            names++;
            if (kind(++i) != T_COMMA) break;
        }
        if (kind(i) == T_LT) {
            const PtxTokenWord t = tk(i + 1);
            uint64_t mag;
            // (a count is a value that no tag expresses: not for a template)
            if (tags || names > 1 || i + 2 >= n || !numeric(t.y >> 16) || (t.y & 0xFFFFu) == 0xFFFFu || kind(i + 2) != T_GT) return false;
            if (ptx_literal_scan(text + t.x, t.y & 0xFFFFu, (uint16_t)(t.y >> 16), &mag) & (PTX_LC_ERR | PTX_LC_GT_U32)) return false;
            count = (uint32_t)mag;
            if (!count) return false;
            i += 3;
        }
        if (one && (count || names > 1)) return false;
        w(((uint32_t)scalar << 8) | (space << 16) | (count ? 1u << 24 : 0u));
        w(0);
        w(0);
        if (initial && !count && kind(i) == T_EQ) {
            Operand o;
            i++;
            if (tags || operand(i, o) != 1 || o.form != F_IMM) return false;
            w(1);
            w(1u + o.kind);
            w((uint32_t)o.bits);
            w((uint32_t)(o.bits >> 32));
        } else {
            w(0);
        }
        if (kind(i) != T_SEMI || i + 1 != n || nw > cap) return false;
        const uint32_t total = nw;
        nw = at;
        w(count ? 1u : 0u);
        w(count);
        w(names);
        nw = total;
        return true;
    }
    PTX_HD static uint32_t space_of(uint32_t k) {
        switch (k) {
        case T_DOT_REG: return StateSpace_Reg;
        case T_MOD_local: return StateSpace_Local;
        case T_MOD_param: return StateSpace_Param;
        case T_MOD_global: return StateSpace_Global;
        case T_MOD_const: return StateSpace_Const;
        case T_MOD_shared: return StateSpace_Shared;
        default: return 0xFFu;
        }
    }
    // a unit inside a function, at this depth of scopes
    PTX_HD bool statement(uint32_t depth) {
        const uint32_t k = kind(0);
        if (n == 1 && (k == T_LBRACE || k == T_RBRACE)) {
            w(k == T_LBRACE ? U_BLOCK_OPEN : depth == 1 ? U_FUNC_END : U_BLOCK_CLOSE);
            return cap != 0;
        }
        if (n == 2 && kind(1) == T_COLON) {
            if (!ident(0)) return false;
            w((uint32_t)U_LABEL | (2u << 8));
            span(0);
            return nw <= cap;
        }
        const uint32_t space = space_of(k);
        if (space == 0xFFu) return instruction();
        w(0);
        if (!variables(1, space, space == StateSpace_Global || space == StateSpace_Const, false)) return false;
        words[0] = (uint32_t)U_VAR | ((nw - 1) << 8);
        return true;
    }
    bool is_func = false;
    // a unit outside of functions
    PTX_HD bool directive() {
        uint32_t i = 0, link = 0;
        for (;; i++) {
            const uint32_t k = kind(i);
            if (k == T_DOT_EXTERN) link |= 1;
            else if (k == T_DOT_VISIBLE) link |= 2;
            else if (k == T_MOD_weak) link |= 4;
            else break;
        }
        if (kind(i) == T_DOT_ENTRY) return is_func = kernel_header(i, link);
        const uint32_t space = space_of(kind(i));
        if (space != StateSpace_Global && space != StateSpace_Const && space != StateSpace_Shared) return false;
        nw = 1;
        w(tk(0).x, PTX_TAG_START << 8);
        w(link);
        if (!variables(i + 1, space, space != StateSpace_Shared, true)) return false;
        words[0] = (uint32_t)U_MODVAR | ((nw - 1) << 8);
        if (tags) tags[0] = 0;
        return true;
    }
    // [linking words] .entry (token i) name ( .param .type name, ... ) {
    PTX_HD bool kernel_header(uint32_t i, uint32_t link) {
        if (!ident(i + 1) || kind(i + 2) != T_LPAREN) return false;
        name_tok = i + 1;
        i += 3;
        nw = 8;
        n_inputs = 0;
        if (kind(i) != T_RPAREN) {
            for (;;) {
                const int scalar = scalar_of(kind(i + 1));
                if (kind(i) != T_MOD_param || scalar < 0 || !ident(i + 2)) return false;
                w(((uint32_t)scalar << 8) | ((uint32_t)StateSpace_Param << 16));
                w(0);
                w(0);
                w(0);
                span(i + 2);
                n_inputs++;
                const uint32_t k = kind(i + 3);
                i += 4;
                if (k == T_RPAREN) break;
                if (k != T_COMMA) return false;
            }
        } else {
            i++;
        }
        if (kind(i) != T_LBRACE || i + 1 != n || nw > cap) return false;
        const PtxTokenWord nm = tk(name_tok);
        const uint32_t total = nw;
        nw = 0;
        w((uint32_t)U_FUNC | ((total - 1) << 8));
        w(link | FUNC_IS_KERNEL | FUNC_HAS_BODY);
        w(nm.x);
        w(nm.y & 0xFFFFu);
        w(0);
        w(n_inputs);
        w(PTX_ABSENT);
        w(tk(0).x);
        nw = total;
        return true;
    }
};
