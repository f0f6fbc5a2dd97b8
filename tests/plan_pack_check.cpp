/* Test driver for tests/test_plan_pack_cpu.py: compiles the ghost fill of
 * each mesh named on the command line (<prefix>.cfg, <prefix>.desc), packs
 * it for the device and expands the pairs again: every list must hold the
 * operations of its kind in program order, each once, and where ghost rows run
 * along k (meshes of several blocks, named after "--") most must be joined.
 * Then a program of its own at the last block a face key holds. */
#include "../fornaxamr_b200/csrc/fx_plan.h"

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

struct Lists { /* cell copies, other cell ops, face copies, other face ops, cell-field ops */
    std::vector<Row> l[5];
};

/* the program's wave; face copies of blocks beyond a key go with the others */
Lists of_program(const FxProgram &g, int w)
{
    Lists r;
    for (int q = g.cell_begin[w]; q < g.cell_begin[w + 1]; ++q) {
        r.l[g.cell_ops[q].type == FX_GOP_COPY ? 0 : 1].push_back(row(0, g.cell_ops[q]));
    }
    for (int q = g.face_begin[w]; q < g.face_begin[w + 1]; ++q) {
        const FxGop &o = g.face_ops[q];
        const bool key = o.type == FX_FOP_COPY && (o.dst >> 15) < 43690 && (o.src >> 15) < 43690;
        r.l[key ? 2 : 3].push_back(row(1, o));
    }
    for (int q = g.b_begin[w]; q < g.b_begin[w + 1]; ++q) r.l[4].push_back(row(g.b_ops[q]));
    return r;
}

Lists of_packed(const FxPacked &k, int w, bool &same)
{
    Lists r;
    for (int q = k.begin[0][w]; q < k.begin[0][w + 1]; ++q) {
        const FxPair &c = k.cp[q];
        for (int h = 0; h < (c.dst < 0 ? 1 : 2); ++h) {
            r.l[0].push_back(row(0, FxGop{(c.dst & 0x7fffffff) + h, c.src + h, 0, FX_GOP_COPY}));
        }
    }
    for (int q = k.begin[1][w]; q < k.begin[1][w + 1]; ++q) r.l[1].push_back(row(0, k.cg[q]));
    for (int q = k.begin[2][w]; q < k.begin[2][w + 1]; ++q) {
        const FxPair &c = k.fp[q];
        const int D = c.dst & 0x7fffffff, S = c.src, dir = (D >> 14) % 3;
        same = same && dir == (S >> 14) % 3;
        for (int h = 0; h < (c.dst < 0 ? 1 : 2); ++h) {
            r.l[2].push_back(row(1, FxGop{(D >> 14) / 3 << 15 | ((D & 16383) + h), (S >> 14) / 3 << 15 | ((S & 16383) + h),
                dir, FX_FOP_COPY}));
        }
    }
    for (int q = k.begin[3][w]; q < k.begin[3][w + 1]; ++q) r.l[3].push_back(row(1, k.fg[q]));
    for (int q = k.begin[4][w]; q < k.begin[4][w + 1]; ++q) {
        for (int h = 0; h < k.b[q].pad; ++h) {
            FxBop o = k.b[q];
            o.dst += h;
            for (int &f : o.f) f += h;
            r.l[4].push_back(row(o));
        }
    }
    return r;
}

/* the same lists; n: operations per list */
bool check(const FxProgram &g, const FxPacked &k, size_t n[5])
{
    bool same = true;
    for (int w = 0; w < g.nwaves(); ++w) {
        const Lists a = of_program(g, w), b = of_packed(k, w, same);
        for (int l = 0; l < 5; ++l) {
            same = same && a.l[l] == b.l[l];
            n[l] += a.l[l].size();
        }
    }
    return same;
}

/* faces of blocks 43689 (the last a key holds) and 43690, as source and as
 * destination: pairs, a pair cut by a block or a direction, odd ends */
bool last_key()
{
    FxProgram g;
    const int blocks[4][2] = {{43689, 43689}, {43689, 43690}, {43690, 43689}, {43690, 43690}};
    for (const int *b : {blocks[0], blocks[1], blocks[2], blocks[3]}) {
        for (int d = 0; d < 3; ++d) {
            for (int f = 8397; f < 8400; ++f) g.face_ops.push_back(FxGop{b[0] << 15 | f, b[1] << 15 | (f - 40), d, FX_FOP_COPY});
            g.face_ops.push_back(FxGop{b[0] << 15 | 20, b[1] << 15 | 60, d, FX_FOP_RESTRICT});
        }
    }
    g.cell_begin = g.b_begin = {0, 0};
    g.face_begin = {0, (int)g.face_ops.size()};
    FxPacked k;
    fx_pack_program(g, k);
    size_t n[5] = {0, 0, 0, 0, 0};
    const bool ok = check(g, k, n) && n[2] == 9 && k.fp.size() == 6 && k.fg.size() == 39;
    printf("last key: %zu + %zu entries: %s\n", k.fp.size(), k.fg.size(), ok ? "same" : "DIFFERENT");
    return ok;
}

} // namespace

int main(int argc, char **argv)
{
    int bad = last_key() ? 0 : 1;
    bool joined = false;
    for (int i = 1; i < argc; ++i) {
        const std::string p = argv[i];
        if (p == "--") {
            joined = true;
            continue;
        }
        const std::vector<fx_config> cfg = load<fx_config>(p + ".cfg");
        const std::vector<fx_block_desc> d = load<fx_block_desc>(p + ".desc");
        FxPlan plan;
        std::string err;
        if (cfg.empty() || !fx_build_plan(cfg[0], (int)d.size(), d.data(), plan, &err)) {
            printf("%s: no plan %s\n", p.c_str(), err.c_str());
            return 2;
        }
        FxPacked k;
        fx_pack_program(plan.ghost, k);
        size_t n[5] = {0, 0, 0, 0, 0};
        bool ok = check(plan.ghost, k, n) && n[0] + n[1] > 0;
        /* share of the operations that sit in an entry of two */
        auto share = [](size_t ops, size_t entries) { return ops ? 2.0 * (double)(ops - entries) / (double)ops : 1.0; };
        const double c = share(n[0], k.cp.size()), f = share(n[2], k.fp.size()), b = share(n[4], k.b.size());
        if (joined) ok = ok && c > 0.85 && f > 0.85 && b > 0.5;
        printf("%s: %zu cell and %zu face copies, %zu cell fields (joined %.2f, %.2f, %.2f), %zu and %zu other entries: %s\n",
            p.c_str(), n[0], n[2], n[4], c, f, b, n[1], n[3], ok ? "same" : "DIFFERENT");
        bad += ok ? 0 : 1;
    }
    return bad;
}
