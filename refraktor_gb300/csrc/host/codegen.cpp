#include "codegen.h"

#include <map>
#include <set>
#include <sstream>

namespace rfk {

namespace {

std::string indent(const std::string& s, int n) {
    std::string pad(n * 4, ' '), out;
    size_t st = 0;
    while (st < s.size()) {
        size_t e = s.find('\n', st);
        if (e == std::string::npos) e = s.size();
        std::string line = s.substr(st, e - st);
        if (!line.empty()) out += pad + line;
        out += "\n";
        st = e + 1;
    }
    return out;
}

struct emitter {
    const flamedb& db;
    std::ostringstream fn;       // xform functions
    std::ostringstream precalc;  // body of rfk_precalc

    // Emits one xform function; `base` is the offset of its weight.
    xform_info xform_fn(const xform& xf, size_t base, int id) {
        xform_info info;
        info.base = base;
        fn << "RFK_FN R rfk_xf_" << id << "(V2& pt, R& col, const PT* RFK_RESTRICT P, Rng& rng) {\n";
        fn << "    V2 in = pt;\n";
        size_t off = base + 4;
        for (size_t li = 0; li < xf.vchain.size(); li++) {
            const vlink& vl = xf.vchain[li];
            const size_t aff = off;
            fn << "    { // vlink " << li << "\n";
            info.affines++;
            fn << "        const R aff_a = P[" << aff << "], aff_d = P[" << aff + 1 << "], aff_b = P[" << aff + 2
               << "], aff_e = P[" << aff + 3 << "], aff_c = P[" << aff + 4 << "], aff_f = P[" << aff + 5 << "];\n";
            fn << "        (void)aff_a; (void)aff_b; (void)aff_c; (void)aff_d; (void)aff_e; (void)aff_f;\n";
            // affine as flame.tpl:10-14 (fma order)
            fn << "        V2 p = fl_vec2(fl_fma(aff_a, in.x, fl_fma(aff_b, in.y, aff_c)), "
                  "fl_fma(aff_d, in.x, fl_fma(aff_e, in.y, aff_f)));\n";
            fn << "        V2 r_ = fl_vec2(R(0), R(0));\n";
            off += 6;
            std::set<std::string> direct;
            for (auto& [vn, _] : vl.variations) {
                const auto& def = db.get_variation(vn);
                for (auto& c : def.apply_usage.commons) direct.insert(c);
            }
            for (auto& cn : db.common_closure(direct)) {
                dsl::emit_env cenv;
                cenv.variation = "common." + cn;
                fn << "        const R c_" << cn << " = " << dsl::emit_expression(db.common_ast(cn), cenv) << ";\n";
            }
            std::ostringstream pc;  // precalc statements for this vlink
            for (auto& [vn, vd] : vl.variations) {
                const auto& def = db.get_variation(vn);
                const size_t v0 = off;
                auto plain = def.plain_params();
                auto pre = def.precalc_params();
                if (plain.size() != vd.params.size() || pre.size() != vd.precalc_count)
                    throw format_error("genome parameters of '" + vn + "' do not match the variation database");
                dsl::emit_env env;
                env.variation = vn;
                env.aff_prefix = "aff_";
                for (size_t i = 0; i < plain.size(); i++) env.param_expr[plain[i]] = "P_" + plain[i];
                for (size_t i = 0; i < pre.size(); i++) env.param_expr[pre[i]] = "P_" + pre[i];
                fn << "        { // " << vn << "\n";
                fn << "            const R w_ = P[" << v0 << "];\n";
                for (size_t i = 0; i < plain.size(); i++)
                    fn << "            const R P_" << plain[i] << " = P[" << v0 + 1 + i << "]; (void)P_" << plain[i] << ";\n";
                for (size_t i = 0; i < pre.size(); i++)
                    fn << "            const R P_" << pre[i] << " = P[" << v0 + 1 + plain.size() + i << "]; (void)P_" << pre[i] << ";\n";
                // a zero-weight variation (padding, or a union kernel's slot
                // that this flame does not use) adds nothing and draws no
                // random numbers; skipping it also keeps 0 * inf out of the sum
                fn << "            if (w_ != R(0)) {\n";
                fn << indent(dsl::emit_body(*def.apply_ast, env), 4);
                fn << "            }\n";
                fn << "        }\n";
                info.rand_calls += def.apply_usage.rand_calls;
                info.sfu_ops += def.apply_usage.sfu_ops;

                if (def.precalc_ast) {
                    dsl::emit_env penv;
                    penv.variation = vn;
                    penv.precalc = true;
                    for (size_t i = 0; i < plain.size(); i++) penv.param_expr[plain[i]] = "P[" + std::to_string(v0 + 1 + i) + "]";
                    for (size_t i = 0; i < pre.size(); i++)
                        penv.param_expr[pre[i]] = "P[" + std::to_string(v0 + 1 + plain.size() + i) + "]";
                    pc << "    { // " << vn << " precalc\n";
                    pc << "        const R w_ = P[" << v0 << "]; (void)w_;\n";
                    pc << indent(dsl::emit_body(*def.precalc_ast, penv), 2);
                    pc << "    }\n";
                }
                off += 1 + plain.size() + pre.size();
            }
            fn << "        in = r_;\n";
            fn << "    }\n";
            if (!pc.str().empty()) {
                precalc << "  { // xform " << id << " vlink " << li << "\n";
                precalc << "    const R aff_a = P[" << aff << "], aff_d = P[" << aff + 1 << "], aff_b = P[" << aff + 2
                        << "], aff_e = P[" << aff + 3 << "], aff_c = P[" << aff + 4 << "], aff_f = P[" << aff + 5 << "];\n";
                precalc << "    (void)aff_a; (void)aff_b; (void)aff_c; (void)aff_d; (void)aff_e; (void)aff_f;\n";
                precalc << pc.str();
                precalc << "  }\n";
            }
        }
        fn << "    pt = in;\n";
        // INTERP(in.z, color, color_speed) = in.z * (1 - cs) + color * cs
        fn << "    col = col * (R(1) - P[" << base + 2 << "]) + P[" << base + 1 << "] * P[" << base + 2 << "];\n";
        fn << "    return P[" << base + 3 << "];\n";
        fn << "}\n\n";
        end = off;
        return info;
    }
    size_t end = 0;

    // One function for all standard xforms (see shared_layout): `X` is an
    // xform's block in shared memory.
    void shared_fn(std::ostringstream& out, const std::vector<std::string>& names) const {
        out << "RFK_FN R rfk_xf_shared(V2& pt, R& col, const PT* RFK_RESTRICT X, Rng& rng) {\n";
        out << "    const rfk_u32 live = __float_as_uint(X[0]);\n";
        out << "    const R aff_a = X[4], aff_d = X[5], aff_b = X[6], aff_e = X[7], aff_c = X[8], aff_f = X[9];\n";
        out << "    (void)aff_a; (void)aff_b; (void)aff_c; (void)aff_d; (void)aff_e; (void)aff_f;\n";
        out << "    V2 p = fl_vec2(fl_fma(aff_a, pt.x, fl_fma(aff_b, pt.y, aff_c)), "
               "fl_fma(aff_d, pt.x, fl_fma(aff_e, pt.y, aff_f)));\n";
        out << "    V2 r_ = fl_vec2(R(0), R(0));\n";
        // a common value is evaluated when a live variation reads it
        std::map<std::string, unsigned> readers;
        std::set<std::string> direct;
        for (size_t v = 0; v < names.size(); v++) {
            const auto& use = db.get_variation(names[v]).apply_usage.commons;
            for (auto& c : db.common_closure(std::set<std::string>(use.begin(), use.end()))) {
                readers[c] |= 1u << v;
                direct.insert(c);
            }
        }
        for (auto& cn : db.common_closure(direct)) {
            dsl::emit_env cenv;
            cenv.variation = "common." + cn;
            out << "    R c_" << cn << " = R(0);\n    if (live & " << readers[cn] << "u) c_" << cn << " = "
                << dsl::emit_expression(db.common_ast(cn), cenv) << ";\n";
        }
        // a loop over the live bits with a switch, instead of a test for each variation,
        // is 13% slower
        size_t off = 10;
        for (size_t v = 0; v < names.size(); v++) {
            const auto& def = db.get_variation(names[v]);
            dsl::emit_env env;
            env.variation = names[v];
            env.aff_prefix = "aff_";
            out << "    if (live & " << (1u << v) << "u) { // " << names[v] << "\n";
            out << "        const R w_ = X[" << off++ << "];\n";
            for (auto& ps : {def.plain_params(), def.precalc_params()})
                for (auto& pn : ps) {
                    env.param_expr[pn] = "P_" + pn;
                    out << "        const R P_" << pn << " = X[" << off++ << "]; (void)P_" << pn << ";\n";
                }
            out << indent(dsl::emit_body(*def.apply_ast, env), 2);
            out << "    }\n";
        }
        out << "    pt = r_;\n";
        out << "    col = col * (R(1) - X[2]) + X[1] * X[2];\n";
        out << "    return X[3];\n}\n\n";
    }
};

// A union-of-variations kernel repeats the code of nearly every variation in
// every xform, more than the instruction cache holds while the warps of a block
// run different xforms: half of its time goes into instruction fetch. From 72
// bodies on (an xform's variations, added up over the standard xforms of one vlink
// each) these share one function instead, and each xform's parameters are laid out
// alike in shared memory:
//   live mask (bit v: the weight of the union's variation v is not 0), colour,
//   colour speed, opacity, affine (6), then per variation its weight, parameters
//   and precalculated parameters (0 where the xform lacks it).
// G iterations/s of rfk_bin with a function per xform and with the shared one
// (xforms x variations each of a union; 8 chains per thread, and by default):
//   24 bodies   12 x 2 of 12   91.6 79.7   96.4 88.4     4 x 6 of 6    89.7 86.9   94.9 95.1
//   42 to 56     6 x 7 of 14   77.7 70.0   78.6 73.5     4 x 14        61.6 59.8   62.2 63.7
//   64 to 70    16 x 4 of 8    88.6 84.7   91.4 91.0    10 x 7 of 14   71.1 69.6   75.3 72.9
//   72          12 x 6 of 12   71.6 73.6   74.7 77.6     6 x 12        68.8 68.5   68.4 73.8
//   80          16 x 5 of 10   75.8 78.4   79.7 81.7     8 x 10        70.5 72.1   72.1 77.5
//   84 to 112   12 x 7 of 14   57.8 68.0   63.5 70.7    16 x 7 of 14   38.8 67.3   37.4 70.0
//   168         12 x 14        24.3 57.5   23.7 61.5
// So 16 or 64 aligned flames of 12 xforms (118 and 158 bodies: 62.1 ms of rfk_bin_batch
// with the first, 72.1 with a function per xform) and the denoiser's sets share one; a
// flame of its own, with one to three variations per xform, keeps a function per xform
// with compile-time offsets. Returns the union's names, empty if not shared.
std::vector<std::string> shared_layout(const flamedb& db, const flame& f, size_t& stride) {
    std::map<std::string, const vardata*> all;
    size_t bodies = 0;
    for (auto& xf : f.xforms) {
        if (xf.vchain.size() != 1) return {};
        for (auto& [vn, vd] : xf.vchain[0].variations) {
            all[vn] = &vd;
            bodies++;
        }
    }
    if (all.size() > 32 || bodies < 72) return {};  // 32 bits of the mask, so three xforms or more
    stride = 10;
    std::vector<std::string> names;
    for (auto& [vn, vd] : all) {
        const auto& def = db.get_variation(vn);
        names.push_back(vn);
        stride += 1 + def.plain_params().size() + def.precalc_params().size();
    }
    stride |= 1;  // odd: the xforms' blocks start in different banks
    if (stride * f.xforms.size() > shared_block_floats) return {};
    return names;
}

}  // namespace

generated_flame generate_flame_code(const flamedb& db, const flame& f) {
    generated_flame g;
    if (f.xforms.empty()) throw format_error("flame has no xforms");
    if (f.xforms.size() > 254) throw format_error("too many xforms");
    for (auto& xf : f.xforms)
        if (xf.vchain.empty()) throw format_error("xform has an empty vchain");
    g.size_reals = f.size_reals();
    g.num_xforms = f.xforms.size();
    g.has_final = f.final_xform.has_value();
    g.chaos = f.chaos.has_value();
    g.affine_indices = f.affine_indices();

    emitter em{db};
    size_t off = 13 + (g.chaos ? g.num_xforms * (g.num_xforms + 1) : 0);
    for (size_t i = 0; i < f.xforms.size(); i++) {
        g.xforms.push_back(em.xform_fn(f.xforms[i], off, (int)i));
        off = em.end;
    }
    if (f.final_xform) {
        g.xforms.push_back(em.xform_fn(*f.final_xform, off, (int)g.num_xforms));
        off = em.end;
    }
    if (off != g.size_reals) throw format_error("internal: packed layout mismatch");

    std::ostringstream s;
    s << "// generated for structure " << f.structure_key() << "\n";
    s << "#ifndef RFK_PARAM_T\n#define RFK_PARAM_T float\n#endif\n";
    s << "typedef RFK_PARAM_T PT;\n";
    s << "#define RFK_NX " << g.num_xforms << "\n";
    s << "#define RFK_HAS_FINAL " << (g.has_final ? 1 : 0) << "\n";
    s << "#define RFK_CHAOS " << (g.chaos ? 1 : 0) << "\n";
    s << "#define RFK_SIZE_REALS " << g.size_reals << "\n";
    s << "#define RFK_NUM_AFFINES " << g.affine_indices.size() << "\n";
    s << "#ifdef RFK_HOST_TWIN\nstatic const unsigned\n#else\n__constant__ unsigned\n#endif\n";
    s << "rfk_affine_idx[RFK_NUM_AFFINES] = {";
    for (size_t i = 0; i < g.affine_indices.size(); i++) s << (i ? ", " : "") << g.affine_indices[i];
    s << "};\n";
    s << "#ifdef RFK_HOST_TWIN\nstatic const unsigned\n#else\n__constant__ unsigned\n#endif\n";
    s << "rfk_xf_base[" << g.xforms.size() << "] = {";
    for (size_t i = 0; i < g.xforms.size(); i++) s << (i ? ", " : "") << g.xforms[i].base;
    s << "};\n\n";
    size_t stride = 0;
    const std::vector<std::string> names = shared_layout(db, f, stride);
    g.shared = !names.empty();
    s << "#define RFK_SHARED " << (g.shared ? 1 : 0) << "\n";
    if (g.shared) {
        s << "#ifndef RFK_HOST_TWIN\n#define RFK_SX_STRIDE " << stride << "\n#define RFK_SX_VARS " << names.size() << "\n";
        // source of each float of the shared-memory blocks in the packed reals
        // (-1: none), and of each variation's weight in a block
        s << "__device__ const short rfk_sx_src[RFK_NX * RFK_SX_STRIDE] = {";
        std::vector<size_t> weight_at;
        for (size_t i = 0; i < g.num_xforms; i++) {
            std::vector<long> row = {-1, (long)g.xforms[i].base + 1, (long)g.xforms[i].base + 2, (long)g.xforms[i].base + 3};
            size_t at = g.xforms[i].base + 4;
            for (int j = 0; j < 6; j++) row.push_back((long)at++);
            weight_at.clear();
            const auto& vars = f.xforms[i].vchain[0].variations;  // sorted by name, as the union is
            for (auto& vn : names) {
                const auto& def = db.get_variation(vn);
                const size_t n = 1 + def.plain_params().size() + def.precalc_params().size();
                weight_at.push_back(row.size());
                const bool has = vars.count(vn) > 0;
                for (size_t j = 0; j < n; j++) row.push_back(has ? (long)at++ : -1);
            }
            row.resize(stride, -1);
            for (size_t j = 0; j < stride; j++) s << (i + j ? ", " : "") << row[j];
        }
        s << "};\n__device__ const short rfk_sx_weight[RFK_SX_VARS] = {";
        for (size_t v = 0; v < weight_at.size(); v++) s << (v ? ", " : "") << weight_at[v];
        s << "};\n";
        em.shared_fn(s, names);
        if (g.has_final) {
            // the final xform keeps its own function
            s << em.fn.str().substr(em.fn.str().rfind("RFK_FN R rfk_xf_"));
        }
        s << "#else\n";
    }
    s << em.fn.str();
    s << "RFK_FN R rfk_dispatch(int k, V2& pt, R& col, const PT* RFK_RESTRICT P, Rng& rng) {\n";
    s << "    switch (k) {\n";
    for (size_t i = 1; i < g.num_xforms; i++) s << "    case " << i << ": return rfk_xf_" << i << "(pt, col, P, rng);\n";
    s << "    default: return rfk_xf_0(pt, col, P, rng);\n";
    s << "    }\n}\n\n";
    if (g.shared) s << "#endif\n";
    if (g.has_final) {
        s << "RFK_FN R rfk_final(V2& pt, R& col, const PT* RFK_RESTRICT P, Rng& rng) {\n";
        s << "    return rfk_xf_" << g.num_xforms << "(pt, col, P, rng);\n}\n\n";
    }
    s << "RFK_FN void rfk_precalc(PT* P, Rng& rng) {\n    (void)P; (void)rng;\n" << em.precalc.str() << "}\n";
    g.source = s.str();
    return g;
}

}  // namespace rfk
