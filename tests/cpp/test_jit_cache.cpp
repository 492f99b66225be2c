// The name of a run-time compiled set's cache file follows everything that its
// cubin is made from (sbf_jit.cpp is included for its internals).
#include "sbf_jit.cpp"

#include <cstdio>
#include <set>

namespace sbf {
bool alphabet_geometry(int, uint32_t*, uint32_t*) { return false; }
}  // namespace sbf

int main() {
    using namespace sbf;
    const JitConfig protein{12, 10, 6, 4, SBF_ALPHABET_PROTEIN, 5, 1};
    const Program base = program_of(protein, "sm_100a");
    const std::string name = cache_file(protein, base, 12, 9);
    if (name != cache_file(protein, program_of(protein, "sm_100a"), 12, 9)) return 1;
    std::set<std::string> names{name};
    size_t n = 1;
    auto differs = [&](const JitConfig& c, const Program& p, int major, int minor) {
        names.insert(cache_file(c, p, major, minor));
        ++n;
    };
    for (size_t v = 0; v < 6; ++v) {  // another kernel in the place of one
        Program p = base;
        p.exprs[v] = p.exprs[v ^ 1];
        differs(protein, p, 12, 9);
    }
    Program p = base;
    std::swap(p.exprs[0], p.exprs[1]);
    differs(protein, p, 12, 9);
    p = base;
    p.src += "\n";
    differs(protein, p, 12, 9);
    p = base;
    p.opts.push_back("-G");
    differs(protein, p, 12, 9);
    differs(protein, program_of(protein, "sm_103a"), 12, 9);
    differs(protein, base, 13, 9);
    differs(protein, base, 12, 8);
    JitConfig other = protein;
    other.h = 8;
    differs(other, program_of(other, "sm_100a"), 12, 9);
    std::printf("%zu of %zu names\n", names.size(), n);
    return names.size() == n ? 0 : 2;
}
