// Host translation unit of the library: the canonical dump (ptx_dump.h) compiled by the host compiler.
#define PTX_HD
#define PTX_TABLE static const
#include "ptx_ast.h"

// the dump by way of the tree's nodes: records -> ptxast nodes, one statement at a time -> text (malloc'ed)
char* ptxfe_dump_module_tree_impl(const PtxBatchView& v, uint32_t m, size_t* len) {
    ptxast::Module mod;
    ptxast::materialize(v, m, &mod, false);
    ptxdump::Out o;
    // a record word prints as about 18 characters
    o.reserve((size_t)(v.results[m].word_end - v.results[m].word_begin) * 20 + 1024);
    ptxast::print_to(o, v, m, mod);
    return o.release(len);
}
// the error list alone, one per line (malloc'ed)
char* ptxfe_error_list_impl(const PtxBatchView& v, uint32_t m, size_t* len) {
    ptxdump::Out o;
    ptxast::print_error_list(o, v, m);
    return o.release(len);
}
// builds and drops the tree of module m; returns the number of nodes built
uint64_t ptxfe_materialize_impl(const PtxBatchView& v, uint32_t m) {
    ptxast::Module mod;
    ptxast::materialize(v, m, &mod);
    return mod.nodes + mod.directives.size();
}
uint64_t ptxfe_dump_hash_impl(const PtxBatchView& v, uint32_t m, int* status) {
    uint64_t h = 0;
    ptxdump::dump_module(v, m, status, &h);
    return h;
}
