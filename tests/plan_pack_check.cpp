/* Test driver for tests/test_plan_pack_cpu.py: compiles the ghost fill of
 * each mesh named on the command line (<prefix>.cfg, <prefix>.desc), packs
 * it for the device and expands the pairs again: every wave must hold the
 * same operations as before, each once. */
#include "../fornaxamr_b200/csrc/fx_plan.h"

#include <algorithm>
#include <array>
#include <cstdio>
#include <string>
#include <vector>

namespace {

template <class T>
std::vector<T> load(const std::string &path)
{
    std::vector<T> v;
    if (FILE *f = fopen(path.c_str(), "rb")) {
        T x;
        while (fread(&x, sizeof x, 1, f) == 1) v.push_back(x);
        fclose(f);
    }
    return v;
}

using Row = std::array<int, 9>;

Row row(int kind, const FxGop &o) { return Row{kind, o.dst, o.src, o.aux, o.type, 0, 0, 0, 0}; }
Row row(const FxBop &o) { return Row{2, o.dst, o.f[0], o.f[1], o.f[2], o.f[3], o.f[4], o.f[5], 0}; }

} // namespace

int main(int argc, char **argv)
{
    int bad = 0;
    for (int i = 1; i < argc; ++i) {
        const std::string p = argv[i];
        const std::vector<fx_config> cfg = load<fx_config>(p + ".cfg");
        const std::vector<fx_block_desc> d = load<fx_block_desc>(p + ".desc");
        FxPlan plan;
        std::string err;
        if (cfg.empty() || !fx_build_plan(cfg[0], (int)d.size(), d.data(), plan, &err)) {
            printf("%s: no plan %s\n", p.c_str(), err.c_str());
            return 2;
        }
        const FxProgram &g = plan.ghost;
        FxPacked k;
        fx_pack_program(g, k);
        size_t ops = 0, pairs = 0;
        bool same = true;
        for (int w = 0; w < g.nwaves(); ++w) {
            std::vector<Row> a, b;
            for (int q = g.cell_begin[w]; q < g.cell_begin[w + 1]; ++q) a.push_back(row(0, g.cell_ops[q]));
            for (int q = g.face_begin[w]; q < g.face_begin[w + 1]; ++q) a.push_back(row(1, g.face_ops[q]));
            for (int q = g.b_begin[w]; q < g.b_begin[w + 1]; ++q) a.push_back(row(g.b_ops[q]));
            for (int q = k.begin[0][w]; q < k.begin[0][w + 1]; ++q) {
                const FxPair &c = k.cp[q];
                const int dst = c.dst & 0x7fffffff;
                for (int h = 0; h < (c.dst < 0 ? 1 : 2); ++h) b.push_back(row(0, FxGop{dst + h, c.src + h, 0, FX_GOP_COPY}));
            }
            for (int q = k.begin[2][w]; q < k.begin[2][w + 1]; ++q) {
                const FxPair &c = k.fp[q];
                const int D = c.dst & 0x7fffffff, S = c.src, dir = (D >> 14) % 3;
                same = same && dir == (S >> 14) % 3;
                for (int h = 0; h < (c.dst < 0 ? 1 : 2); ++h) {
                    b.push_back(row(1, FxGop{(D >> 14) / 3 << 15 | ((D & 16383) + h), (S >> 14) / 3 << 15 | ((S & 16383) + h),
                        dir, FX_FOP_COPY}));
                }
                pairs += c.dst < 0 ? 0 : 1;
            }
            for (int q = k.begin[4][w]; q < k.begin[4][w + 1]; ++q) {
                for (int h = 0; h < k.b[q].pad; ++h) {
                    FxBop o = k.b[q];
                    o.dst += h;
                    for (int &f : o.f) f += h;
                    b.push_back(row(o));
                }
            }
            for (int q = k.begin[1][w]; q < k.begin[1][w + 1]; ++q) b.push_back(row(0, k.cg[q]));
            for (int q = k.begin[3][w]; q < k.begin[3][w + 1]; ++q) b.push_back(row(1, k.fg[q]));
            std::sort(a.begin(), a.end());
            std::sort(b.begin(), b.end());
            same = same && a == b;
            ops += a.size();
        }
        printf("%s: %zu operations in %zu + %zu copies (%zu face pairs), %zu cell-field and %zu + %zu other entries: %s\n", p.c_str(),
            ops, k.cp.size(), k.fp.size(), pairs, k.b.size(), k.cg.size(), k.fg.size(), same && ops ? "same" : "DIFFERENT");
        bad += same && ops ? 0 : 1;
    }
    return bad;
}
