// Lowers one scheduled kernel (SINK → END → STORE(INDEX(PARAM0, ranges), body)) to CUDA C
// for sm_100a.  What the reference does in codegen/lower.go + codegen/wgsl.go for WGSL, redone
// for a machine with 32-wide warps, shared memory and 128-bit global accesses:
//
//  * index arithmetic is canonicalised first.  The scheduler emits reshape/permute/pad as
//    unsimplified i32 div/mod chains (schedule/index.go:231-293); here every integer node is
//    folded into an affine form over the loop variables using their bounds, so that
//    ((r0*I + r1) / I) % B becomes r0.  Strides recovered this way drive the choice between
//    vector and scalar accesses and the thread layout of reductions;
//  * a kernel without REDUCE becomes one thread per V consecutive outputs with 128-bit loads and
//    stores when alignment is provable, scalar otherwise;
//  * REDUCE nodes (several per kernel are allowed, codegen/lower.go:654-719) are evaluated by
//    groups of L threads: lanes stride the flattened reduce space, partial accumulators are
//    combined by warp shuffles and, across warps, shared memory.  L = 1 reproduces the reference's
//    serial ascending loop exactly;
//  * a long REDUCE feeding few outputs is split over many blocks: each writes its partial to scratch
//    memory, and the last of an output's blocks to arrive combines all of them in a fixed order and
//    applies the epilogue, so results do not depend on scheduling.  A REDUCE over the bound batch is
//    rendered a second time in this form, with the number of parts chosen at each launch;
//  * loads whose index cannot be proven inside the buffer (the guarded load of a PAD,
//    schedule/index.go:101-134) are clamped: WGSL defines out-of-range reads, CUDA does not;
//  * guards that compare a SMALL static range with constants are decided while generating: a
//    convolution reaches the device as a sum of K padded slices, each live for exactly one value of
//    the patch index k (tensor/nn/nn.go:256-276), i.e. K selects per multiply.  A reduce loop over
//    such a range is emitted once per value of the range, an output range of that kind becomes a
//    switch over its values, and in every copy the guards fold to true or false — what is left is the
//    one live slice, a direct convolution with the bounds checks of its padding and no im2col buffer.
//
// Arithmetic follows codegen/wgsl.go:240-447: f16 values use native half add/sub/mul outside
// reductions and are widened to f32 inside an f16 reduction with a single narrowing at the end
// (codegen/lower.go:158-171, 698-716); bf16 lives in 32-bit slots and is truncated at the store;
// reduce identities are 0, 1 and -FLT_MAX; infinite literals clamp to +-FLT_MAX.
#include "codegen.hpp"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <sstream>

namespace anl {

uint64_t structure_hash(const Item& item) {
    if (item.shape_hash) return item.shape_hash;
    uint64_t h = 1469598103934665603ull;
    for (const Node& n : item.nodes) {
        int64_t rec[5] = {n.op, n.dtype, n.flags, (int64_t)n.aux, n.arg};
        h = fnv1a(rec, sizeof rec, h);
        for (int s : n.src) h = fnv1a(&s, sizeof s, h);
    }
    for (const BufDesc& b : item.bufs) {
        int64_t rec[2] = {b.dtype, (int64_t)b.shape.size()};
        h = fnv1a(rec, sizeof rec, h);
        for (int64_t s : b.shape) h = fnv1a(&s, sizeof s, h);
    }
    for (const std::string& s : item.sym_vars) h = fnv1a(s.data(), s.size(), h);
    return item.shape_hash = h;
}

namespace {

enum Cls { CF32, CF16, CINT, CUINT, CBOOL };

Cls dtype_cls(int dt) {
    switch (dt) {
        case DT_F16: return CF16;
        case DT_BOOL: return CBOOL;
        case DT_F32: case DT_BF16: case DT_F64: case DT_VOID: return CF32;
        case DT_U8: case DT_U16: case DT_U32: case DT_U64: return CUINT;
        default: return CINT;
    }
}
const char* cls_ctype(Cls c) {
    switch (c) { case CF32: return "float"; case CF16: return "__half"; case CINT: return "int"; case CUINT: return "unsigned"; default: return "bool"; }
}
const char* buf_ctype(int dt) {
    switch (dtype_cls(dt)) { case CF16: return "__half"; case CF32: return "float"; case CINT: return "int"; default: return "unsigned"; }
}

// ── affine forms over loop variables ────────────────────────────────────────────────────────────
struct Lin {
    int64_t c = 0;
    std::vector<std::pair<int, int64_t>> t;   // (atom, coefficient), sorted by atom
    bool is_const() const { return t.empty(); }
};

struct Atom {
    enum Kind { RANGE, DIV, MOD, OPAQUE } kind = RANGE;
    int node = -1;        // RANGE / OPAQUE: node index
    Lin inner;            // DIV / MOD
    int64_t d = 1;
    int64_t lo = 0, hi = 0;
};

const int64_t UNBOUNDED = (int64_t)1 << 40;

struct Gen {
    const Item& it;
    const CodegenOpts& opts;
    std::string err;

    int n;                                 // nodes
    int sink, end, store, body, dst;
    std::vector<int> loop_ranges;          // node indices, END order, loop axis
    std::vector<int> all_ranges;           // every RANGE node
    std::vector<int> range_slot;           // node → slot or -1
    std::vector<std::vector<bool>> dep;    // node × range slot
    std::vector<bool> widen;
    std::vector<int> reduces;              // REDUCE nodes in node order
    bool has_sym = false;

    // ranges that hold one known value while the code around them is being rendered (enumeration)
    std::map<int, int64_t> fixed_range;
    void fix_range(int r, int64_t v) { fixed_range[r] = v; lin_memo.clear(); }
    void unfix_range(int r) { fixed_range.erase(r); lin_memo.clear(); }

    std::vector<Atom> atoms;
    std::map<std::string, int> atom_key;
    std::vector<int> range_atom;           // node → atom
    std::map<int, Lin> lin_memo;

    explicit Gen(const Item& i, const CodegenOpts& o) : it(i), opts(o) {}

    const Node& N(int i) const { return it.nodes[i]; }
    Cls cls(int i) const { Cls c = dtype_cls(N(i).dtype); return (c == CF16 && widen[i]) ? CF32 : c; }

    bool fail(const std::string& m) { if (err.empty()) err = m; return false; }

    // ── structure ──────────────────────────────────────────────────────────────────────────────
    bool analyse() {
        n = (int)it.nodes.size();
        if (n == 0) return fail("codegen: item has no AST");
        sink = n - 1;
        if (N(sink).op != OP_SINK || N(sink).src.empty()) return fail("codegen: last node is not a SINK");
        end = N(sink).src[0];
        if (N(end).op != OP_END || N(end).src.empty()) return fail("codegen: SINK source is not END");
        store = N(end).src[0];
        if (N(store).op != OP_STORE || N(store).src.size() != 2) return fail("codegen: END source is not STORE");
        dst = N(store).src[0];
        body = N(store).src[1];
        range_slot.assign(n, -1);
        for (int i = 0; i < n; i++)
            if (N(i).op == OP_RANGE) { range_slot[i] = (int)all_ranges.size(); all_ranges.push_back(i); if (N(i).symbolic()) has_sym = true; }
        for (size_t s = 1; s < N(end).src.size(); s++) {
            int r = N(end).src[s];
            if (N(r).op == OP_RANGE && N(r).axis() != 1) loop_ranges.push_back(r);
        }
        int nr = (int)all_ranges.size();
        dep.assign(n, std::vector<bool>(nr, false));
        widen.assign(n, false);
        for (int i = 0; i < n; i++) {
            const Node& nd = N(i);
            if (nd.op == OP_RANGE) dep[i][range_slot[i]] = true;
            for (int s : nd.src) for (int r = 0; r < nr; r++) if (dep[s][r]) dep[i][r] = true;
            if (nd.op == OP_REDUCE) {
                reduces.push_back(i);
                for (size_t s = 1; s < nd.src.size(); s++) if (N(nd.src[s]).op == OP_RANGE) dep[i][range_slot[nd.src[s]]] = false;
            }
        }
        // only nodes reachable from the body matter
        std::vector<bool> live(n, false);
        std::function<void(int)> mark = [&](int i) { if (live[i]) return; live[i] = true; for (int s : N(i).src) mark(s); };
        mark(body);
        std::vector<int> lr;
        for (int r : reduces) if (live[r]) lr.push_back(r);
        reduces = lr;
        std::function<void(int)> mw = [&](int i) {
            if (widen[i]) return;
            widen[i] = true;
            if (N(i).op == OP_INDEX) return;
            for (int s : N(i).src) mw(s);
        };
        for (int r : reduces) if (N(r).dtype == DT_F16) mw(N(r).src[0]);
        // atoms for ranges
        range_atom.assign(n, -1);
        for (int r : all_ranges) {
            Atom a; a.kind = Atom::RANGE; a.node = r; a.lo = 0;
            a.hi = N(r).symbolic() ? UNBOUNDED : std::max<int64_t>(N(r).arg - 1, 0);
            range_atom[r] = (int)atoms.size();
            atoms.push_back(a);
        }
        return true;
    }

    // ── guards decided at generation time ─────────────────────────────────────────────────────
    std::set<int> enum_reduce;              // REDUCE nodes whose single small range is emitted value by value
    std::vector<int> enum_out;              // small output ranges turned into a switch over their values

    // Which ranges an integer comparison reads once its operands are in canonical affine form (the
    // scheduler's reshape chains mention every range of the kernel; (n*7056 + hw*9 + k) % 9 is k).
    // False when something other than ranges decides it.
    bool guard_ranges(int i, std::vector<bool>& reads) {
        const Node& nd = N(i);
        if ((nd.op != OP_CMPLT && nd.op != OP_CMPEQ && nd.op != OP_CMPNE) || !is_live(i)) return false;
        if (!is_intlike(nd.src[0]) || !is_intlike(nd.src[1])) return false;
        Lin d = ladd(lin(nd.src[0]), lin(nd.src[1]), -1);
        std::function<bool(const Lin&)> only_ranges = [&](const Lin& l) {
            for (auto& t : l.t) { const Atom& a = atoms[t.first]; if (a.kind == Atom::OPAQUE) return false; if (a.kind != Atom::RANGE && !only_ranges(a.inner)) return false; }
            return true;
        };
        if (!only_ranges(d)) return false;
        reads.assign(all_ranges.size(), false);
        bool any = false;
        for (size_t r = 0; r < all_ranges.size(); r++) if (lin_reads(d, all_ranges[r])) { reads[r] = true; any = true; }
        return any;
    }
    // Fraction of the value combinations of `ranges` for which guard `g` holds (1 where it does not fold).
    double guard_truth(int g, const std::vector<int>& ranges) {
        int64_t combos = 1;
        for (int r : ranges) combos *= N(r).arg;
        int64_t yes = 0;
        const Node& nd = N(g);
        for (int64_t cs = 0; cs < combos; cs++) {
            int64_t rem = cs;
            for (int e = (int)ranges.size() - 1; e >= 0; e--) { fixed_range[ranges[e]] = rem % N(ranges[e]).arg; rem /= N(ranges[e]).arg; }
            lin_memo.clear();
            Lin d = ladd(lin(nd.src[0]), lin(nd.src[1]), -1);
            bool t = true;
            if (d.is_const()) t = nd.op == OP_CMPLT ? d.c < 0 : nd.op == OP_CMPEQ ? d.c == 0 : d.c != 0;
            if (t) yes++;
        }
        for (int r : ranges) fixed_range.erase(r);
        lin_memo.clear();
        return (double)yes / (double)combos;
    }

    // Decides which small ranges are enumerated.  A set of ranges qualifies when at least four guards
    // read exactly that set and, averaged over the set's value combinations, those guards hold less
    // than three times out of four: they select slices (a patch index equal to a constant) instead of
    // merely trimming a border (a padded row, true almost everywhere).
    void plan_enumeration() {
        enum_reduce.clear(); enum_out.clear();
        if (has_sym || opts.debug_bounds) return;
        // A gather without a REDUCE (the scatter-back of a convolution's patches: a sum of one padded slice per channel
        // and tap) is enumerated over its output ranges the same way: 72 clamped loads an output became 9, 15.3 us
        // for 32 x 8 x 14 x 14 outputs became 5.8.
        const size_t nr = all_ranges.size();
        std::map<std::vector<int>, std::vector<int>> by_set;       // ranges read (node indices, sorted) -> guards
        std::vector<bool> reads;
        for (int i = 0; i < n; i++) {
            if (!guard_ranges(i, reads)) continue;
            std::vector<int> key; int64_t prod = 1; bool ok = true;
            for (size_t r = 0; r < nr; r++) if (reads[r]) {
                const Node& rn = N(all_ranges[r]);
                if (rn.symbolic() || rn.arg < 2 || rn.arg > 128) { ok = false; break; }
                key.push_back(all_ranges[r]); prod *= rn.arg;
            }
            if (ok && !key.empty() && prod <= 128) by_set[key].push_back(i);
        }
        struct Cand { std::vector<int> ranges; double score, frac; };
        std::vector<Cand> outs;
        for (auto& kv : by_set) {
            if (kv.second.size() < 4) continue;
            double frac = 0;
            for (int g : kv.second) frac += guard_truth(g, kv.first);
            frac /= (double)kv.second.size();
            if (frac > 0.75) continue;
            // a single reduce range: value-by-value loop of the REDUCE that owns it
            if (kv.first.size() == 1 && N(kv.first[0]).axis() == 1) {
                for (int red : reduces) {
                    std::vector<int> rr;
                    for (size_t s2 = 1; s2 < N(red).src.size(); s2++) if (N(N(red).src[s2]).op == OP_RANGE) rr.push_back(N(red).src[s2]);
                    if (rr.size() == 1 && rr[0] == kv.first[0]) enum_reduce.insert(red);
                }
                continue;
            }
            bool all_out = true;
            for (int r : kv.first) if (std::find(loop_ranges.begin(), loop_ranges.end(), r) == loop_ranges.end()) all_out = false;
            if (all_out) outs.push_back(Cand{kv.first, (double)kv.second.size() * (1.0 - frac), frac});
        }
        std::sort(outs.begin(), outs.end(), [](const Cand& x, const Cand& y) { return x.score > y.score; });
        std::set<int> chosen; int64_t prod = 1;
        double off = 0;            // share of the guards that a case decides against; a slice has two
        for (auto& c : outs) {
            int64_t p2 = prod;
            for (int r : c.ranges) if (!chosen.count(r)) p2 *= N(r).arg;
            if (p2 > 128) continue;
            for (int r : c.ranges) chosen.insert(r);
            prod = p2; off = std::max(off, 1.0 - c.frac);
        }
        // Without a REDUCE the switch has to be paid for by the terms that it leaves out, and neighbouring threads must share
        // the case, or a warp walks through all of them.  16384 x p x 8, a concatenation of p pieces, in us, guarded loads against
        // switch: p = 4 6.1 / 8.2, 8 10.2 / 10.2, 16 20.5 / 14.3, 64 199 / 51; with the pieces along the last range 65536 x 2p
        // 6.1 / 10.2, 10.2 / 16.4, 18.4 / 43, 201 / 168; with 4 elements behind it a scatter of 72 terms 7.4 / 8.2.
        if (reduces.empty()) {
            int64_t behind = 1;
            for (size_t r = loop_ranges.size(); r-- > 0 && !chosen.count(loop_ranges[r]);) behind *= N(loop_ranges[r]).arg;
            int loads = 0;
            for (int i = 0; i < n; i++) if (N(i).op == OP_INDEX && i != dst && is_live(i)) loads++;
            if (loads * off < 6.0 || behind < 8) return;
        }
        for (int r : loop_ranges) if (chosen.count(r)) enum_out.push_back(r);
    }

    // forget what was rendered inside reduce loop `red` (ctx == red), so that it can be rendered again
    void forget_loop(int red) {
        for (auto it = memo.begin(); it != memo.end();) { if (it->first.second == red) it = memo.erase(it); else ++it; }
        loop[red] = Block();
    }

    bool depends_on_reduce(int node, int red) const {
        const Node& r = N(red);
        for (size_t s = 1; s < r.src.size(); s++) {
            int rn = r.src[s];
            if (N(rn).op == OP_RANGE && dep[node][range_slot[rn]]) return true;
        }
        return false;
    }

    // ── Lin algebra ────────────────────────────────────────────────────────────────────────────
    static Lin lconst(int64_t c) { Lin l; l.c = c; return l; }
    Lin latom(int a) const { Lin l; l.t.push_back({a, 1}); return l; }
    static Lin ladd(const Lin& a, const Lin& b, int64_t sb = 1) {
        Lin r; r.c = a.c + sb * b.c;
        size_t i = 0, j = 0;
        while (i < a.t.size() || j < b.t.size()) {
            if (j == b.t.size() || (i < a.t.size() && a.t[i].first < b.t[j].first)) r.t.push_back(a.t[i++]);
            else if (i == a.t.size() || b.t[j].first < a.t[i].first) { r.t.push_back({b.t[j].first, sb * b.t[j].second}); j++; }
            else { int64_t c = a.t[i].second + sb * b.t[j].second; if (c) r.t.push_back({a.t[i].first, c}); i++; j++; }
        }
        return r;
    }
    static Lin lscale(const Lin& a, int64_t k) {
        Lin r; if (k == 0) return r;
        r.c = a.c * k; for (auto& p : a.t) r.t.push_back({p.first, p.second * k});
        return r;
    }
    int64_t llo(const Lin& l) const {
        int64_t v = l.c;
        for (auto& p : l.t) { int64_t b = p.second > 0 ? atoms[p.first].lo : atoms[p.first].hi; if (std::llabs(b) >= UNBOUNDED) return p.second > 0 ? (b < 0 ? -UNBOUNDED : v) : -UNBOUNDED; v += p.second * b; }
        return v;
    }
    int64_t lhi(const Lin& l) const {
        int64_t v = l.c;
        for (auto& p : l.t) { int64_t b = p.second > 0 ? atoms[p.first].hi : atoms[p.first].lo; if (std::llabs(b) >= UNBOUNDED) return UNBOUNDED; v += p.second * b; }
        return v;
    }
    std::string lkey(const Lin& l) const {
        std::ostringstream o; o << l.c;
        for (auto& p : l.t) o << "+" << p.second << "*a" << p.first;
        return o.str();
    }
    int make_atom(Atom::Kind k, const Lin& inner, int64_t d, int64_t lo, int64_t hi, int node = -1) {
        std::ostringstream key;
        key << (int)k << ":" << node << ":" << d << ":" << lkey(inner);
        auto f = atom_key.find(key.str());
        if (f != atom_key.end()) return f->second;
        Atom a; a.kind = k; a.inner = inner; a.d = d; a.lo = lo; a.hi = hi; a.node = node;
        atoms.push_back(a);
        atom_key[key.str()] = (int)atoms.size() - 1;
        return (int)atoms.size() - 1;
    }
    // split e = d*q + r with every coefficient of q*d a multiple of d and 0 <= const(r) < d
    void split(const Lin& e, int64_t d, Lin& q, Lin& r) const {
        q = Lin(); r = Lin();
        int64_t cq = e.c / d, cr = e.c % d;
        if (cr < 0) { cr += d; cq -= 1; }
        q.c = cq; r.c = cr;
        for (auto& p : e.t) {
            if (p.second % d == 0) q.t.push_back({p.first, p.second / d});
            else r.t.push_back(p);
        }
    }
    Lin ldiv(const Lin& e, int64_t d) {
        if (d == 1) return e;
        if (e.is_const()) return lconst(e.c / d);
        int64_t lo = llo(e), hi = lhi(e);
        if (d <= 0 || lo < 0) return latom(make_atom(Atom::DIV, e, d, -UNBOUNDED, UNBOUNDED));
        Lin q, r; split(e, d, q, r);
        if (r.is_const()) return q;                       // r.c in [0,d)
        int64_t rlo = llo(r), rhi = lhi(r);
        if (rlo >= 0 && rhi < d) return q;
        if (rlo >= 0) return ladd(q, latom(make_atom(Atom::DIV, r, d, rlo / d, rhi >= UNBOUNDED ? UNBOUNDED : rhi / d)));
        return latom(make_atom(Atom::DIV, e, d, lo / d, hi >= UNBOUNDED ? UNBOUNDED : hi / d));
    }
    Lin lmod(const Lin& e, int64_t m) {
        if (m == 1) return lconst(0);
        if (e.is_const() && m > 0) return lconst(e.c % m);
        int64_t lo = llo(e), hi = lhi(e);
        if (m <= 0 || lo < 0) return latom(make_atom(Atom::MOD, e, m, -UNBOUNDED, UNBOUNDED));
        if (hi < m) return e;
        Lin q, r; split(e, m, q, r);
        if (r.is_const()) return lconst(r.c);
        int64_t rlo = llo(r), rhi = lhi(r);
        if (rlo >= 0 && rhi < m) return r;
        if (rlo >= 0) return latom(make_atom(Atom::MOD, r, m, 0, std::min(m - 1, rhi)));
        return latom(make_atom(Atom::MOD, e, m, 0, m - 1));
    }

    bool is_intlike(int i) const { Cls c = dtype_cls(N(i).dtype); return c == CINT || c == CUINT; }

    Lin lin(int i) {
        auto f = lin_memo.find(i);
        if (f != lin_memo.end()) return f->second;
        const Node& nd = N(i);
        Lin r;
        switch (nd.op) {
            case OP_CONST: r = lconst(nd.arg); break;
            case OP_RANGE: { auto fx = fixed_range.find(i); r = fx != fixed_range.end() ? lconst(fx->second) : latom(range_atom[i]); break; }
            case OP_ADD: r = ladd(lin(nd.src[0]), lin(nd.src[1])); break;
            case OP_SUB: r = ladd(lin(nd.src[0]), lin(nd.src[1]), -1); break;
            case OP_NEG: r = lscale(lin(nd.src[0]), -1); break;
            case OP_MUL: {
                Lin a = lin(nd.src[0]), b = lin(nd.src[1]);
                if (b.is_const()) r = lscale(a, b.c);
                else if (a.is_const()) r = lscale(b, a.c);
                else r = latom(make_atom(Atom::OPAQUE, Lin(), 1, -UNBOUNDED, UNBOUNDED, i));
                break;
            }
            case OP_IDIV: {
                Lin b = lin(nd.src[1]);
                if (b.is_const() && b.c > 0) r = ldiv(lin(nd.src[0]), b.c);
                else r = latom(make_atom(Atom::OPAQUE, Lin(), 1, -UNBOUNDED, UNBOUNDED, i));
                break;
            }
            case OP_MOD: {
                Lin b = lin(nd.src[1]);
                if (b.is_const() && b.c > 0) r = lmod(lin(nd.src[0]), b.c);
                else r = latom(make_atom(Atom::OPAQUE, Lin(), 1, -UNBOUNDED, UNBOUNDED, i));
                break;
            }
            default: r = latom(make_atom(Atom::OPAQUE, Lin(), 1, -UNBOUNDED, UNBOUNDED, i)); break;
        }
        lin_memo[i] = r;
        return r;
    }

    // does the affine form read loop variable `range_node`, directly or through an atom?
    bool lin_reads(const Lin& l, int range_node) const {
        for (auto& p : l.t) {
            const Atom& a = atoms[p.first];
            if (a.kind == Atom::RANGE) { if (a.node == range_node) return true; }
            else if (a.kind == Atom::OPAQUE) { if (dep[a.node][range_slot[range_node]]) return true; }
            else if (lin_reads(a.inner, range_node)) return true;
        }
        return false;
    }
    // coefficient of a loop variable when it appears only as a direct term; ok=false otherwise
    int64_t lin_coef(const Lin& l, int range_node, bool& ok) const {
        int64_t c = 0; ok = true;
        for (auto& p : l.t) {
            const Atom& a = atoms[p.first];
            if (a.kind == Atom::RANGE && a.node == range_node) c = p.second;
            else if (a.kind != Atom::RANGE) {
                Lin one; one.t.push_back({p.first, 1});
                if (lin_reads(one, range_node)) ok = false;
            }
        }
        return c;
    }

    // ── flat load index ────────────────────────────────────────────────────────────────────────
    Lin flat_index(int index_node) {
        const Node& nd = N(index_node);
        int p = (int)N(nd.src[0]).arg;
        int ndim = (int)nd.src.size() - 1;
        if (ndim == 0) return lconst(0);
        if (ndim == 1) return lin(nd.src[1]);
        const std::vector<int64_t>& sh = it.bufs[p].shape;
        std::vector<int64_t> st(ndim, 1);
        for (int d = ndim - 2; d >= 0; d--) st[d] = (d + 1 < (int)sh.size()) ? st[d + 1] * (sh[d + 1] ? sh[d + 1] : 1) : 1;
        Lin r;
        for (int d = 0; d < ndim; d++) r = ladd(r, lscale(lin(nd.src[1 + d]), st[d]));
        return r;
    }
    bool in_bounds(const Lin& f, int param) const {
        const BufDesc& b = it.bufs[param];
        int64_t lo = llo(f), hi = lhi(f);
        if (!b.symbolic()) return lo >= 0 && hi < b.elems(0);
        // symbolic outermost dim: need coef(sym range) == trailing and the rest inside one row
        int64_t tr = b.trailing();
        Lin rest; rest.c = f.c; bool found = false;
        for (auto& p : f.t) {
            const Atom& a = atoms[p.first];
            if (a.kind == Atom::RANGE && N(a.node).symbolic()) { if (p.second != tr) return false; found = true; }
            else rest.t.push_back(p);
        }
        return found && llo(rest) >= 0 && lhi(rest) < tr;
    }

    // ── emission ───────────────────────────────────────────────────────────────────────────────
    struct Block { std::string code; int indent = 1; };
    Block top;                              // statements outside reduce loops
    std::map<int, Block> loop;              // REDUCE node → statements inside its loop
    std::map<std::pair<int, int>, std::string> memo;   // (node, ctx) → expression
    int vec_range = -1;                     // loop variable unrolled by the vector path, or -1
    std::map<int, std::string> vec_load;    // INDEX node → array name holding V preloaded values
    // A row's reduction and then a sweep over it in one kernel (build_rowbcast): with wide loads or an unroll count on the
    // reduction the compiler leaves the sweep, which is the longer part, without its own unrolling (100000 values in one
    // block 37 us as it is, 80 with wide loads; 4096 rows of 9000 90 and 116).
    bool row_broadcast = false;
    int split_parts = 1;                    // blocks an output (-1: counted at launch)
    bool split_mode = false;                // every output's REDUCE is shared by SPLIT blocks (build_reduce)
    int reduce_vec = 1;                     // consecutive elements a lane takes per trip of the innermost reduce range
    std::string reduce_combine_mode;        // set by the kernel builder
    int lanes = 1, touts = 1, threads = 256; bool rc_layout = true;

    // One reduce loop that serves several outputs (build_side_by_side): reduce_expr leaves its parts here instead of in `top`
    struct SideBySide { bool on = false, ok = true; std::string tag, decl, head, body, acc; int reds = 0; } side;

    std::vector<std::pair<Lin, int>>* loads_seen = nullptr;      // index and element size of every load rendered, while thread_order counts them
    Block prelude;                          // vector path: statements that must precede the unrolled loop
    Block* cur_top = nullptr;
    std::map<int, std::vector<bool>> atom_dep_memo;

    Block& T() { return cur_top ? *cur_top : top; }

    void stmt(int ctx, const std::string& s) {
        Block& b = ctx < 0 ? (cur_top ? *cur_top : top) : loop[ctx];
        b.code += std::string((ctx < 0 ? 1 : 2) * 2, ' ') + s + "\n";
    }

    // loop variables an atom reads, as a bitset over range slots
    const std::vector<bool>& atom_dep(int ai) {
        auto f = atom_dep_memo.find(ai);
        if (f != atom_dep_memo.end()) return f->second;
        std::vector<bool> d(all_ranges.size(), false);
        const Atom& a = atoms[ai];
        if (a.kind == Atom::RANGE) d[range_slot[a.node]] = true;
        else if (a.kind == Atom::OPAQUE) d = dep[a.node];
        else for (auto& p : a.inner.t) { const std::vector<bool>& s = atom_dep(p.first); for (size_t r = 0; r < d.size(); r++) if (s[r]) d[r] = true; }
        return atom_dep_memo[ai] = d;
    }
    bool atom_in_reduce(int ai, int red) {
        const std::vector<bool>& d = atom_dep(ai);
        const Node& r = N(red);
        for (size_t s = 1; s < r.src.size(); s++) if (N(r.src[s]).op == OP_RANGE && d[range_slot[r.src[s]]]) return true;
        return false;
    }
    // DIV / MOD atoms get a named temporary in the outermost context that can hold them
    std::string atom_name(int ai, int ctx) {
        if (ctx >= 0 && !atom_in_reduce(ai, ctx)) ctx = -1;
        auto key = std::make_pair(-(ai + 1), ctx);
        auto f = memo.find(key);
        if (f != memo.end()) return f->second;
        const Atom& a = atoms[ai];
        std::string name = "a" + std::to_string(ai);
        stmt(ctx, "const int " + name + " = " + render(a.inner, ctx) + (a.kind == Atom::DIV ? " / " : " % ") + std::to_string(a.d) + ";");
        memo[key] = name;
        return name;
    }

    std::string range_name(int r) const {
        auto fx = fixed_range.find(r);
        if (fx != fixed_range.end()) return std::to_string(fx->second);
        std::string s = "r" + std::to_string(N(r).aux);
        return r == vec_range ? "(" + s + " + u)" : s;
    }

    std::string render(const Lin& l, int ctx) {
        if (l.is_const()) return l.c < 0 ? "(" + std::to_string(l.c) + ")" : std::to_string(l.c);
        std::string s = "(";
        bool first = true;
        for (auto& p : l.t) {
            const Atom& a = atoms[p.first];
            std::string v;
            switch (a.kind) {
                case Atom::RANGE: v = range_name(a.node); break;
                case Atom::DIV: case Atom::MOD: v = atom_name(p.first, ctx); break;
                case Atom::OPAQUE: v = opaque_int(a.node, ctx); break;
            }
            int64_t c = p.second;
            if (!first) s += c < 0 ? " - " : " + ";
            else if (c < 0) s += "-";
            int64_t ac = std::llabs(c);
            s += ac == 1 ? v : v + " * " + std::to_string(ac);
            first = false;
        }
        if (l.c > 0) s += " + " + std::to_string(l.c);
        else if (l.c < 0) s += " - " + std::to_string(-l.c);
        return s + ")";
    }

    static std::string flit(double d) {
        float f = (float)d;
        if (std::isnan(f)) return "__int_as_float(0x7fc00000)";
        if (std::isinf(f)) return f < 0 ? "__int_as_float(0xff7fffff)" : "__int_as_float(0x7f7fffff)";
        char b[64]; std::snprintf(b, sizeof b, "%af", (double)f);
        return std::string(b);
    }
    static bool is_zero_lit(const std::string& e) { return e == "0x0p+0f" || e == "__float2half_rn(0x0p+0f)"; }
    // x * 1.0 is x bit for bit in IEEE arithmetic (the gradient of a sum multiplies by ones)
    bool is_float_one(int i) const {
        const Node& nd = N(i);
        if (nd.op != OP_CONST || !dt_is_float(nd.dtype)) return false;
        double d; std::memcpy(&d, &nd.arg, 8);
        return d == 1.0;
    }

    std::string const_lit(int i) {
        const Node& nd = N(i);
        if (dt_is_float(nd.dtype)) {
            double d; std::memcpy(&d, &nd.arg, 8);
            bool f16 = nd.dtype == DT_F16;
            if (f16 && std::isinf(d)) d = d < 0 ? -65504.0 : 65504.0;
            std::string f = flit(d);
            return (f16 && !widen[i]) ? "__float2half_rn(" + f + ")" : f;
        }
        if (nd.dtype == DT_BOOL) return nd.arg ? "true" : "false";
        if (nd.arg == INT32_MIN) return "(-2147483647 - 1)";
        return nd.arg < 0 ? "(" + std::to_string(nd.arg) + ")" : std::to_string(nd.arg);
    }

    // integer node that the affine engine could not absorb: plain C on its operands
    std::string opaque_int(int i, int ctx) {
        if (ctx >= 0 && !depends_on_reduce(i, ctx)) ctx = -1;
        auto key = std::make_pair(i, ctx);
        auto f = memo.find(key);
        if (f != memo.end()) return f->second;
        const Node& nd = N(i);
        std::string e;
        auto a = [&](int k) { return val(nd.src[k], ctx); };
        switch (nd.op) {
            case OP_MUL: e = "(" + a(0) + " * " + a(1) + ")"; break;
            case OP_IDIV: e = "idiv_(" + a(0) + ", " + a(1) + ")"; break;
            case OP_MOD: e = "imod_(" + a(0) + ", " + a(1) + ")"; break;
            case OP_MAX: e = "max(" + a(0) + ", " + a(1) + ")"; break;
            case OP_SHL: e = "(" + a(0) + " << (" + a(1) + " & 31))"; break;
            case OP_SHR: e = "(" + a(0) + " >> (" + a(1) + " & 31))"; break;
            case OP_AND: e = "(" + a(0) + " & " + a(1) + ")"; break;
            case OP_OR: e = "(" + a(0) + " | " + a(1) + ")"; break;
            case OP_XOR: e = "(" + a(0) + " ^ " + a(1) + ")"; break;
            case OP_WHERE: e = "(" + a(0) + " ? " + a(1) + " : " + a(2) + ")"; break;
            case OP_MULACC: e = "(" + a(0) + " + (" + a(1) + " * " + a(2) + "))"; break;
            case OP_CAST: case OP_BITCAST: e = cast_expr(i, ctx); break;
            case OP_INDEX: e = load_expr(i, ctx); break;
            case OP_REDUCE: e = reduce_expr(i); break;
            default: fail("codegen: unhandled integer op " + std::to_string(nd.op)); e = "0"; break;
        }
        std::string name = "t" + std::to_string(i);
        stmt(ctx, std::string("const ") + cls_ctype(cls(i)) + " " + name + " = " + e + ";");
        memo[key] = name;
        return name;
    }

    std::string to_float(int src, const std::string& e) {
        switch (cls(src)) { case CF32: return e; case CF16: return "__half2float(" + e + ")"; case CBOOL: return "(" + e + " ? 1.0f : 0.0f)"; default: return "(float)(" + e + ")"; }
    }
    std::string cast_expr(int i, int ctx) {
        const Node& nd = N(i);
        int s = nd.src[0];
        std::string e = val(s, ctx);
        Cls to = cls(i), from = cls(s);
        if (nd.op == OP_BITCAST) {
            if (to == from) return e;
            if (to == CF32 && (from == CINT || from == CUINT)) return "__int_as_float((int)" + e + ")";
            if ((to == CINT || to == CUINT) && from == CF32) return std::string("(") + cls_ctype(to) + ")__float_as_int(" + e + ")";
            fail("codegen: unsupported bitcast"); return "0";
        }
        if (to == from) return e;
        switch (to) {
            case CF32: return to_float(s, e);
            case CF16: return "__float2half_rn(" + to_float(s, e) + ")";
            case CBOOL: return from == CF16 ? "(__half2float(" + e + ") != 0.0f)" : from == CF32 ? "(" + e + " != 0.0f)" : "(" + e + " != 0)";
            case CINT: return from == CF16 ? "(int)__half2float(" + e + ")" : "(int)(" + e + ")";
            default: return from == CF16 ? "(unsigned)__half2float(" + e + ")" : "(unsigned)(" + e + ")";
        }
    }

    // Row chain whose rows fit the registers of a block (render_row_chain): every sweep over the row is `row_chunks`
    // chunks of `row_vec` elements a lane, and row-contiguous operands are read from register arrays.
    int64_t row_len = 0;                             // 0: not in this form
    int row_vec = 1, row_chunks = 0;
    std::map<int, std::string> row_reg;              // INDEX node -> register array holding this lane's elements of the row
    int* row_slot = nullptr;                         // next shared-memory segment for a reduction over the row

    // Rows whose length is no multiple of the width start anywhere in a 16-byte group: the chunks are then laid from the
    // group the row starts in (`shift` elements before it), and every element says for itself whether it is the row's.
    bool row_shifted = false;

    // the elements of one sweep as a loop nest around a body that sees them as variable `rn`; u indexes the registers
    std::string row_open(const std::string& rn, bool guarded) const {
        const std::string V = std::to_string(row_vec), C = std::to_string(row_len);
        std::string s = "  _Pragma(\"unroll\") for (int c = 0; c < " + std::to_string(row_chunks) + "; c++) {\n    const int cb = (c * LANES + lane) * " + V + (row_shifted ? " - shift" : "") + ";\n";
        if (!row_exact() && !row_shifted) s += "    const bool live = cb < " + C + ";\n";
        if (guarded && !row_exact() && !row_shifted) s += "    if (live)\n";
        s += "    _Pragma(\"unroll\") for (int v = 0; v < " + V + "; v++) { const int u = c * " + V + " + v, " + rn + " = cb + v; (void)u; (void)" + rn + ";\n";
        if (row_shifted) s += "    const bool live = (unsigned)" + rn + " < " + C + "u; (void)live;\n";
        if (row_shifted && guarded) s += "    if (!live) continue;\n";
        return s;
    }
    bool row_exact() const { return !row_shifted && row_len == (int64_t)row_chunks * row_vec * lanes; }

    // Is INDEX node i, under sweep variable `sweep`, element (row, sweep) of a row-contiguous f32 or f16 buffer?
    bool row_contiguous(int i, int sweep, int64_t C) {
        const Node& nd = N(i);
        if (nd.op != OP_INDEX || N(nd.src[0]).op != OP_PARAM || loop_ranges.empty()) return false;
        const int p = (int)N(nd.src[0]).arg;
        if (p <= 0 || p >= (int)it.bufs.size() || chain_subst.count(p) || it.bufs[p].symbolic()) return false;
        const int dt = it.bufs[p].dtype;
        if ((dt != DT_F32 && dt != DT_F16) || dtype_cls(nd.dtype) == CBOOL) return false;
        Lin f = flat_index(i);
        if (f.c != 0 || !in_bounds(f, p)) return false;
        int64_t cr = N(loop_ranges[0]).arg == 1 ? C : 0, cs = 0;
        for (auto& t : f.t) {
            const Atom& a = atoms[t.first];
            if (a.kind != Atom::RANGE) return false;
            if (a.node == loop_ranges[0]) cr = t.second;
            else if (a.node == sweep) cs = t.second;
            else return false;
        }
        return cr == C && cs == 1;
    }
    // Is parameter p read at element (row, sweep) of a dense matrix of C columns and nowhere else?
    bool reads_own_row(int p, int64_t C) {
        for (int i = 0; i < n; i++) {
            if (N(i).op != OP_INDEX || i == dst || !is_live(i) || N(N(i).src[0]).op != OP_PARAM || N(N(i).src[0]).arg != p) continue;
            const Lin f = flat_index(i);
            bool row = false, sweep = false;
            for (auto& t : f.t) {
                const Atom& a = atoms[t.first];
                if (a.kind != Atom::RANGE) return false;
                if (a.node == loop_ranges[0] && t.second == C) row = true;
                else if (a.node != loop_ranges[0] && t.second == 1 && !N(a.node).symbolic() && N(a.node).arg == C) sweep = true;
                else return false;
            }
            if (f.c != 0 || f.t.size() != 2 || !row || !sweep) return false;
        }
        return true;
    }
    // The sweeps of a chain stage all run over the same static extent C, one range each: C, and the row-contiguous loads
    // with the sweep variable they follow; 0 when the stage is not of this form, -1 when it sweeps nothing.
    int64_t row_extent(std::vector<int>& loads) {
        int64_t C = -1;
        std::vector<int> sweeps;
        for (int r : reduces) {
            std::vector<int> rr;
            for (size_t k = 1; k < N(r).src.size(); k++) if (N(N(r).src[k]).op == OP_RANGE) rr.push_back(N(r).src[k]);
            if (rr.size() != 1) return 0;
            sweeps.push_back(rr[0]);
        }
        if (loop_ranges.size() > 2) return 0;
        if (loop_ranges.size() == 2) sweeps.push_back(loop_ranges[1]);
        for (int w : sweeps) {
            if (N(w).symbolic() || (C >= 0 && N(w).arg != C)) return 0;
            C = N(w).arg;
        }
        for (int i = 0; i < n; i++) {
            if (N(i).op != OP_INDEX || i == dst || !is_live(i)) continue;
            for (int w : sweeps) if (row_contiguous(i, w, C)) { loads.push_back(i); break; }
        }
        return C;
    }
    // does the sweep body below `root` load anything but registers?
    bool row_loads_memory(int root, int sweep) {
        std::vector<int> stack{root};
        std::set<int> seen;
        while (!stack.empty()) {
            int j = stack.back(); stack.pop_back();
            if (!seen.insert(j).second || !dep[j][range_slot[sweep]]) continue;
            if (N(j).op == OP_INDEX) { if (!row_reg.count(j)) return true; continue; }
            for (int c : N(j).src) stack.push_back(c);
        }
        return false;
    }

    bool unroll_short_loops = false;
    int chain_vec = 1;
    std::string dp = "data";                         // name prefix of the buffer pointers
    std::map<int, std::string> chain_subst;          // row chain: parameter → register holding this row's value

    // Row-chain stages with chain_vec > 1: INDEX nodes below `root` (nested reductions excluded) that
    // sweep `sweep` with unit stride and whose address is provably a multiple of chain_vec elements
    // when the sweep variable is (16-byte aligned bases, every other term a multiple of chain_vec).
    // Each gets one wide load per chunk into a small array; load_expr then hands out array[u].
    // Returns the declarations + loads, written for a scope in which the sweep variable holds the
    // chunk's first index.
    std::string chain_wide_loads(int root, int sweep, int ctx) {
        std::string code;
        if (chain_vec <= 1 || opts.debug_bounds) return code;
        std::vector<int> stack{root}, seen_nodes;
        std::set<int> seen;
        while (!stack.empty()) {
            int j = stack.back(); stack.pop_back();
            if (!seen.insert(j).second) continue;
            const Node& nd = N(j);
            if (nd.op == OP_REDUCE && j != root) continue;
            if (nd.op == OP_INDEX) { seen_nodes.push_back(j); continue; }
            for (int c : nd.src) stack.push_back(c);
        }
        std::sort(seen_nodes.begin(), seen_nodes.end());
        const std::string V = std::to_string(chain_vec);
        for (int j : seen_nodes) {
            const Node& nd = N(j);
            if (N(nd.src[0]).op != OP_PARAM || !dep[j][range_slot[sweep]]) continue;
            int p = (int)N(nd.src[0]).arg;
            if (p <= 0 || p >= (int)it.bufs.size() || chain_subst.count(p)) continue;
            Cls bc = dtype_cls(it.bufs[p].dtype);
            const bool widens = bc == CF16 && cls(j) == CF32;        // f16 storage inside an f16 reduction
            if ((bc != cls(j) && !widens) || (bc != CF32 && bc != CF16) || dtype_cls(nd.dtype) == CBOOL) continue;
            Lin f = flat_index(j);
            if (!in_bounds(f, p) || f.c % chain_vec != 0) continue;
            bool ok = true;
            for (auto& t : f.t) {
                const Atom& a = atoms[t.first];
                if (a.kind != Atom::RANGE) { ok = false; break; }
                if (a.node == sweep ? t.second != 1 : t.second % chain_vec != 0) { ok = false; break; }
            }
            bool cok; if (!ok || lin_coef(f, sweep, cok) != 1 || !cok) continue;
            const std::string arr = "vl" + std::to_string(j) + "_" + std::to_string(ctx < 0 ? 0 : ctx), bt = buf_ctype(it.bufs[p].dtype);
            const std::string raw = widens ? arr + "h" : arr;
            code += "    " + bt + " " + raw + "[" + V + "];\n";
            code += "    ldv_<" + bt + ", " + V + ">(" + dp + std::to_string(p) + " + " + render(f, ctx) + ", " + raw + ");\n";
            if (widens) code += "    float " + arr + "[" + V + "];\n    _Pragma(\"unroll\") for (int u = 0; u < " + V + "; u++) " + arr + "[u] = __half2float(" + raw + "[u]);\n";
            vec_load[j] = arr;
        }
        return code;
    }

    std::string load_expr(int i, int ctx) {
        if (vec_load.count(i)) return vec_load[i] + "[u]";
        const Node& nd = N(i);
        auto rg = row_reg.find(i);
        if (rg != row_reg.end()) {
            const std::string e = rg->second + "[u]";
            const Cls bc = dtype_cls(it.bufs[(int)N(nd.src[0]).arg].dtype), want = cls(i);
            return bc == CF16 && want == CF32 ? "__half2float(" + e + ")" : bc == CF32 && want == CF16 ? "__float2half_rn(" + e + ")" : e;
        }
        if (N(nd.src[0]).op != OP_PARAM) { fail("codegen: INDEX of a non-parameter"); return "0"; }
        int p = (int)N(nd.src[0]).arg;
        if (p < 0 || p >= (int)it.bufs.size()) { fail("codegen: PARAM number out of range"); return "0"; }
        Lin f = flat_index(i);
        if (loads_seen) loads_seen->push_back({f, dt_storage_bytes(it.bufs[p].dtype)});
        auto cs = chain_subst.find(p);
        if (cs != chain_subst.end()) {
            // produced by an earlier stage of the same row chain: only this row's element is available
            bool row_only = f.c == 0 && f.t.size() == 1 && f.t[0].second == 1 && atoms[f.t[0].first].kind == Atom::RANGE &&
                            !loop_ranges.empty() && atoms[f.t[0].first].node == loop_ranges[0];
            if (!row_only) { fail("chain: a stage reads another row of an earlier stage's output"); return "0"; }
            std::string e = cs->second;
            Cls bc = dtype_cls(it.bufs[p].dtype), want = cls(i);
            if (dtype_cls(nd.dtype) == CBOOL) return "(" + e + " != 0u)";
            if (bc == CF16 && want == CF32) return "__half2float(" + e + ")";
            if (bc == CF32 && want == CF16) return "__float2half_rn(" + e + ")";
            if (bc != want && (want == CINT || want == CUINT)) return std::string("(") + cls_ctype(want) + ")" + e;
            if (bc != want && want == CF32) return "(float)" + e;
            return e;
        }
        std::string idx = render(f, ctx);
        if (opts.debug_bounds || !in_bounds(f, p)) {
            const BufDesc& b = it.bufs[p];
            std::string hi = b.symbolic() ? "(n0 * " + std::to_string(b.trailing()) + " - 1)" : std::to_string(std::max<int64_t>(b.elems(0) - 1, 0));
            idx = "clampi_(" + idx + ", " + hi + ")";
        }
        std::string e = dp + std::to_string(p) + "[" + idx + "]";
        Cls bc = dtype_cls(it.bufs[p].dtype);
        Cls want = cls(i);
        if (dtype_cls(nd.dtype) == CBOOL) return "(" + e + " != 0u)";
        if (bc == CF16 && want == CF32) return "__half2float(" + e + ")";
        if (bc == CF32 && want == CF16) return "__float2half_rn(" + e + ")";
        if (bc != want && (want == CINT || want == CUINT)) return std::string("(") + cls_ctype(want) + ")" + e;
        if (bc != want && want == CF32) return "(float)" + e;
        return e;
    }

    std::string identity(int rop, Cls c) {
        if (c == CF32 || c == CF16) return rop == OP_MUL ? "1.0f" : rop == OP_MAX ? "__int_as_float(0xff7fffff)" : "0.0f";
        if (c == CUINT) return rop == OP_MUL ? "1u" : "0u";
        return rop == OP_MUL ? "1" : rop == OP_MAX ? "(-2147483647 - 1)" : "0";
    }
    std::string combine(int rop, Cls c, const std::string& a, const std::string& b) {
        bool f = (c == CF32 || c == CF16);
        switch (rop) {
            case OP_MUL: return "(" + a + " * " + b + ")";
            case OP_MAX: return f ? "fmaxf(" + a + ", " + b + ")" : "max(" + a + ", " + b + ")";
            default: return "(" + a + " + " + b + ")";
        }
    }
    const char* rop_tag(int rop) { return rop == OP_MUL ? "mul" : rop == OP_MAX ? "max" : "add"; }

    // bound of a reduce range as a C expression
    std::string range_bound(int r) { return N(r).symbolic() ? "n0" : std::to_string(N(r).arg); }

    // Elements of the innermost reduce range a lane takes per trip: 8 where every wide load is f16, else 4, else 1.
    // Only where lanes run along the reduce range (RC layout), the range is static and a multiple of the
    // width, and at least one operand then arrives by 128-bit loads.
    int pick_reduce_vec(int red, const std::vector<int>& rr) {
        if (!rc_layout || rr.empty() || unroll_short_loops || row_broadcast || opts.debug_bounds || opts.vector_width == 1 || enum_reduce.count(red)) return 1;
        const int last = rr.back();
        if (N(last).symbolic() || N(last).arg < 64) return 1;
        const int keep = chain_vec;
        const std::map<int, std::string> before = vec_load;
        for (int V : {8, 4}) {
            if (N(last).arg % V) continue;
            // eight wide trips a lane, or (split) what the part count leaves; a shorter loop has all its loads in flight
            // as it is, and keeps the order of its additions
            if (!split_mode && reduce_total(red) < (int64_t)lanes * V * 8) continue;
            chain_vec = V;
            const std::string probe = chain_wide_loads(N(red).src[0], last, red);
            bool any = false, f16 = true;
            for (auto& kv : vec_load) if (!before.count(kv.first)) { any = true; if (dt_storage_bytes(it.bufs[(int)N(N(kv.first).src[0]).arg].dtype) != 2) f16 = false; }
            vec_load = before;
            chain_vec = keep;
            if (any && (V == 4 || f16)) return V;
        }
        return 1;
    }

    // Trips of a reduce loop whose loads the compiler may issue together: eight for a short body, fewer where the
    // copies would bloat the kernel, never more than a lane makes.  The additions stay in order.  Without it each trip
    // waits for its own loads: a column sum over 64 rows by four lanes took 9.2 us (16 dependent trips), now 3.3.  From 32
    // trips on the compiler's own choice is better (65536 x 1024 f32 summed over the rows 178 us eight at a time, 60 so; 8192 x 8192
    // f16 46 and 37), and where the parts are counted at launch a lane makes as many.
    std::string loop_unroll(int red, int64_t terms) {
        const int64_t lines = (int64_t)std::count(loop[red].code.begin(), loop[red].code.end(), '\n');
        if (row_broadcast) return std::string();
        int64_t u = lines <= 12 ? 8 : lines <= 30 ? 4 : lines <= 60 ? 2 : 1;
        if (!enum_out.empty()) u = 1;           // a copy per case already: 72 cases unrolled four times ran 37.7 us instead of 22.6, from instruction memory
        if (terms > 0) while (u > 1 && u * lanes > terms) u /= 2;
        if (split_parts > 1) terms /= split_parts;
        if (terms >= (int64_t)lanes * 32 || split_parts < 0) u = 1;
        return u > 1 ? "_Pragma(\"unroll " + std::to_string(u) + "\") " : std::string();
    }

    std::string reduce_expr(int i) {
        const Node& nd = N(i);
        int rop = (int)nd.aux;
        Cls c = dtype_cls(nd.dtype);
        bool isf = (c == CF32 || c == CF16);
        Cls acc_c = isf ? CF32 : c;
        const char* at = isf ? "float" : cls_ctype(acc_c);
        std::string acc = "acc" + std::to_string(i);
        std::vector<int> rr;
        for (size_t s = 1; s < nd.src.size(); s++) if (N(nd.src[s]).op == OP_RANGE) rr.push_back(nd.src[s]);
        if (side.on) {
            side.acc = acc + side.tag;
            side.decl = std::string("  ") + at + " " + side.acc + " = " + identity(rop, acc_c) + ";\n";
            const std::string e = val(nd.src[0], i), ef = (isf && cls(nd.src[0]) == CF16) ? "__half2float(" + e + ")" : e;
            side.ok = side.ok && ++side.reds == 1 && !rr.empty() && T().code.empty();     // nothing may have been hoisted: the outputs share the text in front
            std::string tot, vars, stride = "1";
            for (int k = (int)rr.size() - 1; k >= 0; k--) {
                const std::string rn = "r" + std::to_string(N(rr[k]).aux), b = range_bound(rr[k]);
                vars += "    const int " + rn + " = " + (k == 0 ? "q / (" + stride + ")" : "(q / (" + stride + ")) % " + b) + "; (void)" + rn + ";\n";
                stride += " * " + b;
                tot = tot.empty() ? b : b + " * " + tot;
            }
            side.head = "  for (int q = RED_BEGIN(" + tot + "); q < RED_END(" + tot + "); q += RED_STEP) {\n" + vars;
            side.body = "    {\n" + loop[i].code + "    " + side.acc + " = " + combine(rop, acc_c, side.acc, ef) + ";\n    }\n";
            return nd.dtype == DT_F16 ? "__float2half_rn(" + side.acc + ")" : side.acc;
        }
        stmt(-1, std::string(at) + " " + acc + " = " + identity(rop, acc_c) + ";");
        {
            if (enum_reduce.count(i) && lanes == 1 && rr.size() == 1) {
                // one copy of the loop body per value of the range: the guards that read it fold away, and
                // so does every term of the body that they switch off
                const int R = rr[0];
                for (int64_t kk = 0; kk < N(R).arg; kk++) {
                    fix_range(R, kk);
                    forget_loop(i);
                    std::string e = val(nd.src[0], i);
                    std::string ef = (isf && cls(nd.src[0]) == CF16) ? "__half2float(" + e + ")" : e;
                    if (rop == OP_ADD && is_zero_lit(e) && loop[i].code.empty()) continue;       // nothing live for this value
                    T().code += "  {   // r" + std::to_string(N(R).aux) + " = " + std::to_string(kk) + "\n" + loop[i].code;
                    T().code += "    " + acc + " = " + combine(rop, acc_c, acc, ef) + ";\n  }\n";
                }
                unfix_range(R);
                forget_loop(i);
                if (nd.dtype == DT_F16) return "__float2half_rn(" + acc + ")";
                return acc;
            }
            if (row_len > 0 && rr.size() == 1) {
                // Row held in registers: the body runs for every element a lane holds, the ones past the end of the row
                // included (their registers are zero), and only what it adds is selected; so that an exponential that
                // several sweeps need is one value to the compiler, not one per branch.
                const std::string e = val(nd.src[0], i);
                const std::string ef = (isf && cls(nd.src[0]) == CF16) ? "__half2float(" + e + ")" : e;
                const bool mem = row_loads_memory(nd.src[0], rr[0]);
                T().code += row_open("r" + std::to_string(N(rr[0]).aux), mem) + loop[i].code;
                const std::string sum = combine(rop, acc_c, acc, ef);
                T().code += "    " + acc + " = " + (mem || row_exact() ? sum : "live ? " + sum + " : " + acc) + ";\n  } }\n";
                stmt(-1, acc + " = row_" + std::string(rop_tag(rop)) + "_" + (isf ? "f" : "i") + "(" + acc + ", red_smem + " + std::to_string(32 * (*row_slot)++) + ");");
                if (nd.dtype == DT_F16) return "__float2half_rn(" + acc + ")";
                return acc;
            }
            // row-chain stage sweeping the row in chunks: the wide loads must be known before the body is rendered
            bool chunked = false;
            std::string wide;
            std::vector<int> wide_nodes;
            if (rr.size() == 1 && unroll_short_loops && chain_vec > 1 && !N(rr[0]).symbolic() &&
                N(rr[0]).arg <= (int64_t)lanes * 32 && N(rr[0]).arg % ((int64_t)lanes * chain_vec) == 0) {
                chunked = true;
                std::map<int, std::string> before = vec_load;
                wide = chain_wide_loads(nd.src[0], rr[0], i);
                for (auto& kv : vec_load) if (!before.count(kv.first)) wide_nodes.push_back(kv.first);
            }
            // elsewhere: the innermost reduce range taken reduce_vec elements at a time where that gives wide loads
            const int rvec = chunked ? 1 : pick_reduce_vec(i, rr);
            if (rvec > 1) {
                std::map<int, std::string> before = vec_load;
                const int keep = chain_vec;
                chain_vec = rvec;
                wide = chain_wide_loads(nd.src[0], rr.back(), i);
                chain_vec = keep;
                for (auto& kv : vec_load) if (!before.count(kv.first)) wide_nodes.push_back(kv.first);
            }
            reduce_vec = rvec;
            std::string e = val(nd.src[0], i);
            for (int j : wide_nodes) vec_load.erase(j);
            std::string ef = (isf && cls(nd.src[0]) == CF16) ? "__half2float(" + e + ")" : e;
            // emit: loop header, hoisted code is already in `top`, then the loop body
            std::string hdr;
            if (rr.empty()) {
                hdr = split_mode ? "if (lane == 0 && part == 0) {" : "if (lane == 0) {";
            } else if (rvec > 1) {
                std::string tot = "(";
                for (size_t k = 0; k < rr.size(); k++) tot += (k ? " * " : "") + range_bound(rr[k]);
                tot += ")";
                const std::string V = std::to_string(rvec);
                hdr = "_Pragma(\"unroll 4\") for (int q = RED_BEGIN_V(" + tot + ", " + V + "); q < RED_END(" + tot + "); q += RED_STEP * " + V + ") {";
            } else if (rr.size() == 1) {
                std::string rn = "r" + std::to_string(N(rr[0]).aux);
                hdr = "for (int " + rn + " = RED_BEGIN(" + range_bound(rr[0]) + "); " + rn + " < RED_END(" + range_bound(rr[0]) + "); " + rn + " += RED_STEP) {";
                bool whole = false;
                // short trip counts are unrolled: the loads of one stage of a row chain can then stay in
                // registers for the next stage instead of being fetched from L1 again
                if (unroll_short_loops && !N(rr[0]).symbolic() && N(rr[0]).arg <= (int64_t)lanes * 32) {
                    whole = true;
                    if (chunked) {
                        // each lane takes chain_vec consecutive elements per trip; unit-stride operands
                        // arrive by one explicit 128-bit load per chunk (the inner declaration of the
                        // sweep variable shadows the chunk's first index the loads are written with)
                        std::string V = std::to_string(chain_vec), nb = range_bound(rr[0]);
                        hdr = "_Pragma(\"unroll\") for (int " + rn + "b = lane * " + V + "; " + rn + "b < " + nb + "; " + rn + "b += LANES * " + V + ") {\n"
                              "    const int " + rn + " = " + rn + "b; (void)" + rn + ";\n" + wide +
                              "  _Pragma(\"unroll\") for (int u = 0; u < " + V + "; u++) { const int " + rn + " = " + rn + "b + u;";
                    } else hdr = "_Pragma(\"unroll\") " + hdr;
                }
                if (!whole) hdr = loop_unroll(i, reduce_total(i)) + hdr;
            } else {
                std::string tot = "(";
                for (size_t k = 0; k < rr.size(); k++) tot += (k ? " * " : "") + range_bound(rr[k]);
                tot += ")";
                hdr = loop_unroll(i, reduce_total(i)) + "for (int q = RED_BEGIN" + tot + "; q < RED_END" + tot + "; q += RED_STEP) {";
            }
            T().code += "  " + hdr + "\n";
            if (rr.size() > 1 || rvec > 1) {
                // decompose q, last range fastest
                std::string stride = "1";
                for (int k = (int)rr.size() - 1; k >= 0; k--) {
                    std::string rn = "r" + std::to_string(N(rr[k]).aux);
                    std::string b = range_bound(rr[k]);
                    T().code += "    const int " + rn + " = " + (k == 0 ? "q / (" + stride + ")" : "(q / (" + stride + ")) % " + b) + "; (void)" + rn + ";\n";
                    stride = stride + " * " + b;
                }
            }
            if (rvec > 1) {
                // the inner declaration shadows the chunk's first index, which the wide loads are written with
                const std::string rn = "r" + std::to_string(N(rr.back()).aux);
                T().code += wide + "    const int " + rn + "b = " + rn + ";\n";
                T().code += "  _Pragma(\"unroll\") for (int u = 0; u < " + std::to_string(rvec) + "; u++) { const int " + rn + " = " + rn + "b + u; (void)" + rn + ";\n";
            }
            T().code += loop[i].code;
            T().code += "    " + acc + " = " + combine(rop, acc_c, acc, ef) + ";\n";
            T().code += chunked || rvec > 1 ? "  } }\n" : "  }\n";
            reduce_vec = std::max(reduce_vec, rvec);
            const std::string tag = std::string(rop_tag(rop)) + "_" + (isf ? "f" : "i");
            if (reduce_combine_mode == "group") stmt(-1, acc + " = group_" + tag + "(" + acc + ", lane, grp, red_smem);");
            if (split_mode) stmt(-1, "if (!join_" + tag + "(" + acc + ", " + identity(rop, acc_c) + ", lane, grp, red_smem, &split_last, scratch, tickets, ob, part, SPLIT, NOB)) return;");
        }
        if (nd.dtype == DT_F16) return "__float2half_rn(" + acc + ")";
        return acc;
    }

    // value of node i as a C expression usable in context ctx (-1 = outside reduce loops)
    std::string val(int i, int ctx) {
        const Node& nd = N(i);
        if (nd.op == OP_CONST) return const_lit(i);
        if (nd.op == OP_RANGE) return range_name(i);
        if (ctx >= 0 && !depends_on_reduce(i, ctx)) ctx = -1;
        Cls c = cls(i);
        if ((c == CINT || c == CUINT) && nd.op != OP_INDEX && nd.op != OP_REDUCE && nd.op != OP_CAST && nd.op != OP_BITCAST && nd.op != OP_WHERE)
            return render(lin(i), ctx);
        if (c == CINT || c == CUINT) return opaque_int(i, ctx);
        auto key = std::make_pair(i, ctx);
        auto f = memo.find(key);
        if (f != memo.end()) return f->second;
        std::string e;
        auto a = [&](int k) { return val(nd.src[k], ctx); };
        auto af = [&](int k) { return to_float(nd.src[k], val(nd.src[k], ctx)); };
        // operand k in this node's own compute class: a node shared between an f16 reduction (where it
        // is evaluated widened) and f16 code outside it is narrowed at the point of use
        auto ac = [&](int k) {
            std::string v = val(nd.src[k], ctx);
            Cls sc = cls(nd.src[k]);
            if (sc == c) return v;
            if (c == CF16 && sc == CF32) return "__float2half_rn(" + v + ")";
            if (c == CF32 && sc == CF16) return "__half2float(" + v + ")";
            return v;
        };
        bool h = (c == CF16);
        auto wrap = [&](const std::string& fexpr) { return h ? "__float2half_rn(" + fexpr + ")" : fexpr; };
        if (c == CBOOL) {
            switch (nd.op) {
                case OP_CMPLT: case OP_CMPNE: case OP_CMPEQ: {
                    int s0 = nd.src[0], s1 = nd.src[1];
                    const char* o = nd.op == OP_CMPLT ? " < " : nd.op == OP_CMPNE ? " != " : " == ";
                    if (is_intlike(s0) && is_intlike(s1)) {
                        Lin d = ladd(lin(s0), lin(s1), -1);     // s0 - s1
                        int64_t lo = llo(d), hi = lhi(d);
                        if (nd.op == OP_CMPLT) { if (hi < 0) return "true"; if (lo >= 0) return "false"; }
                        if (nd.op == OP_CMPNE) { if (hi < 0 || lo > 0) return "true"; if (lo == 0 && hi == 0) return "false"; }
                        if (nd.op == OP_CMPEQ) { if (hi < 0 || lo > 0) return "false"; if (lo == 0 && hi == 0) return "true"; }
                        e = "(" + render(lin(s0), ctx) + o + render(lin(s1), ctx) + ")";
                    } else if (cls(s0) == CF16 || cls(s1) == CF16) e = "(" + af(0) + o + af(1) + ")";
                    else e = "(" + a(0) + o + a(1) + ")";
                    break;
                }
                case OP_AND: { std::string x = a(0), y = a(1); if (x == "false" || y == "false") return "false"; if (x == "true") return y; if (y == "true") return x; e = "(" + x + " && " + y + ")"; break; }
                case OP_OR: { std::string x = a(0), y = a(1); if (x == "true" || y == "true") return "true"; if (x == "false") return y; if (y == "false") return x; e = "(" + x + " || " + y + ")"; break; }
                case OP_XOR: e = "(" + a(0) + " != " + a(1) + ")"; break;
                case OP_WHERE: e = "(" + a(0) + " ? " + a(1) + " : " + a(2) + ")"; break;
                case OP_CAST: case OP_BITCAST: e = cast_expr(i, ctx); break;
                case OP_INDEX: e = load_expr(i, ctx); break;
                default: fail("codegen: unhandled bool op " + std::to_string(nd.op)); return "false";
            }
        } else {
            switch (nd.op) {
                case OP_INDEX: e = load_expr(i, ctx); break;
                case OP_REDUCE: if (ctx >= 0) { fail("codegen: nested REDUCE"); return "0.0f"; } e = reduce_expr(i); break;
                case OP_CAST: case OP_BITCAST: e = cast_expr(i, ctx); break;
                case OP_WHERE: { std::string cnd = a(0); if (cnd == "true") return ac(1); if (cnd == "false") return ac(2); e = "(" + cnd + " ? " + ac(1) + " : " + ac(2) + ")"; break; }
                // one MUFU: results below 2^-126 flush to zero instead of going through exp2f's rescaling
                // for subnormals (absolute difference < 1.2e-38)
                case OP_EXP2: e = h ? "__float2half_rn(ex2_h_(" + af(0) + "))" : "ex2_h_(" + af(0) + ")"; break;
                case OP_LOG2: e = wrap("log2f(" + af(0) + ")"); break;
                case OP_SIN: e = wrap("sinf(" + af(0) + ")"); break;
                case OP_SQRT: e = wrap("sqrtf(" + af(0) + ")"); break;
                case OP_RECIP: e = h ? "__float2half_rn(rcp_h_(" + af(0) + "))" : "__frcp_rn(" + af(0) + ")"; break;
                case OP_TRUNC: e = wrap("truncf(" + af(0) + ")"); break;
                case OP_NEG: e = h ? "__hneg(" + ac(0) + ")" : "(-" + ac(0) + ")"; break;
                case OP_ADD: {
                    // x + 0 where the zero is what a guard folded to (a padded slice that is not live):
                    // the value of x, at worst with the sign of a zero changed
                    std::string x0 = ac(0), x1 = ac(1);
                    if (is_zero_lit(x0)) return x1;
                    if (is_zero_lit(x1)) return x0;
                    e = h ? "__hadd(" + x0 + ", " + x1 + ")" : "(" + x0 + " + " + x1 + ")"; break;
                }
                case OP_SUB: e = h ? "__hsub(" + ac(0) + ", " + ac(1) + ")" : "(" + ac(0) + " - " + ac(1) + ")"; break;
                case OP_MUL:
                    if (is_float_one(nd.src[0]) && cls(nd.src[1]) == c) return ac(1);
                    if (is_float_one(nd.src[1]) && cls(nd.src[0]) == c) return ac(0);
                    e = h ? "__hmul(" + ac(0) + ", " + ac(1) + ")" : "(" + ac(0) + " * " + ac(1) + ")"; break;
                case OP_FDIV: e = wrap("(" + af(0) + " / " + af(1) + ")"); break;
                case OP_MAX: e = h ? "__hmax(" + ac(0) + ", " + ac(1) + ")" : "fmaxf(" + ac(0) + ", " + ac(1) + ")"; break;
                case OP_POW: e = wrap("powf(" + af(0) + ", " + af(1) + ")"); break;
                case OP_MOD: e = wrap("fmodf(" + af(0) + ", " + af(1) + ")"); break;
                case OP_MULACC: e = h ? "__hadd(" + ac(0) + ", __hmul(" + ac(1) + ", " + ac(2) + "))" : "(" + ac(0) + " + (" + ac(1) + " * " + ac(2) + "))"; break;
                default: fail("codegen: unhandled op " + std::to_string(nd.op)); return "0.0f";
            }
        }
        std::string name = "t" + std::to_string(i);
        stmt(ctx, std::string("const ") + cls_ctype(c) + " " + name + " = " + e + ";");
        memo[key] = name;
        return name;
    }

    // ── paired f16 evaluation ────────────────────────────────────────────────────────────────
    // An elementwise kernel whose values are all f16 (or comparisons of f16 values) is evaluated two
    // elements at a time in __half2: every arithmetic instruction then serves two outputs, which is
    // what an instruction-bound GELU needs to get back under the memory roofline.  Each lane
    // computes exactly what the one-element form computes (the *2 intrinsics round per lane, exp2 and
    // the reciprocal go through the same f32 approximations), so the two forms agree bit for bit.
    bool h2 = false;

    bool h2_node_ok(int i, std::vector<char>& seen) {
        if (seen[i]) return seen[i] == 1;
        seen[i] = 1;
        const Node& nd = N(i);
        Cls c = cls(i);
        auto fail_ = [&]() { seen[i] = 2; return false; };
        if (nd.op == OP_CONST) return (nd.dtype == DT_F16 && c == CF16) ? true : fail_();
        if (nd.op == OP_INDEX) {
            if (c != CF16 || N(nd.src[0]).op != OP_PARAM) return fail_();
            int p = (int)N(nd.src[0]).arg;
            if (p < 0 || p >= (int)it.bufs.size() || it.bufs[p].dtype != DT_F16) return fail_();
            return true;                                   // the index subtree is integer code, rendered as usual
        }
        if (c == CF16) {
            switch (nd.op) {
                case OP_NEG: case OP_ADD: case OP_SUB: case OP_MUL: case OP_MAX: case OP_MULACC:
                case OP_EXP2: case OP_LOG2: case OP_SQRT: case OP_RECIP: case OP_SIN: break;
                case OP_WHERE: if (cls(nd.src[0]) != CBOOL) return fail_(); break;
                default: return fail_();
            }
        } else if (c == CBOOL) {
            switch (nd.op) {
                case OP_CMPLT: case OP_CMPNE: case OP_CMPEQ:
                    if (cls(nd.src[0]) != CF16 || cls(nd.src[1]) != CF16) return fail_();
                    break;
                case OP_AND: case OP_OR: case OP_XOR: case OP_WHERE: break;
                default: return fail_();
            }
        } else return fail_();
        for (int sidx : nd.src) if (!h2_node_ok(sidx, seen)) return fail_();
        return true;
    }
    bool h2_eligible(int V) {
        if (V < 2 || (V & 1) || it.bufs[0].dtype != DT_F16 || cls(body) != CF16) return false;
        std::vector<char> seen(n, 0);
        return h2_node_ok(body, seen);
    }

    std::string val_h2(int i) {
        const Node& nd = N(i);
        auto key = std::make_pair(i, -1);
        auto f = memo.find(key);
        if (f != memo.end()) return f->second;
        if (nd.op == OP_CONST) {
            double d; std::memcpy(&d, &nd.arg, 8);
            if (std::isinf(d)) d = d < 0 ? -65504.0 : 65504.0;
            return "__float2half2_rn(" + flit(d) + ")";
        }
        Cls c = cls(i);
        auto a = [&](int k) { return val_h2(nd.src[k]); };
        std::string e;
        switch (nd.op) {
            case OP_INDEX: e = vec_load.count(i) ? vec_load[i] + "[u]" : "__half2half2(" + load_expr(i, -1) + ")"; break;
            case OP_NEG: e = "__hneg2(" + a(0) + ")"; break;
            case OP_ADD: e = "__hadd2(" + a(0) + ", " + a(1) + ")"; break;
            case OP_SUB: e = "__hsub2(" + a(0) + ", " + a(1) + ")"; break;
            case OP_MUL:
                if (is_float_one(nd.src[0])) return a(1);
                if (is_float_one(nd.src[1])) return a(0);
                e = "__hmul2(" + a(0) + ", " + a(1) + ")"; break;
            case OP_MAX: e = "__hmax2(" + a(0) + ", " + a(1) + ")"; break;
            case OP_MULACC: e = "__hadd2(" + a(0) + ", __hmul2(" + a(1) + ", " + a(2) + "))"; break;
            case OP_EXP2: e = "h2_ex2_(" + a(0) + ")"; break;
            case OP_RECIP: e = "h2_rcp_(" + a(0) + ")"; break;
            case OP_LOG2: e = "h2_log2_(" + a(0) + ")"; break;
            case OP_SQRT: e = "h2_sqrt_(" + a(0) + ")"; break;
            case OP_SIN: e = "h2_sin_(" + a(0) + ")"; break;
            case OP_CMPLT: e = "__hlt2_mask(" + a(0) + ", " + a(1) + ")"; break;
            case OP_CMPEQ: e = "__heq2_mask(" + a(0) + ", " + a(1) + ")"; break;
            case OP_CMPNE: e = "__hneu2_mask(" + a(0) + ", " + a(1) + ")"; break;
            case OP_AND: e = "(" + a(0) + " & " + a(1) + ")"; break;
            case OP_OR: e = "(" + a(0) + " | " + a(1) + ")"; break;
            case OP_XOR: e = "(" + a(0) + " ^ " + a(1) + ")"; break;
            case OP_WHERE:
                e = c == CBOOL ? "((" + a(0) + " & " + a(1) + ") | (~" + a(0) + " & " + a(2) + "))" : "h2_sel_(" + a(0) + ", " + a(1) + ", " + a(2) + ")";
                break;
            default: fail("codegen: paired f16 form met op " + std::to_string(nd.op)); return "__float2half2_rn(0.0f)";
        }
        std::string name = "t" + std::to_string(i);
        stmt(-1, std::string("const ") + (c == CBOOL ? "unsigned" : "__half2") + " " + name + " = " + e + ";");
        memo[key] = name;
        return name;
    }

    std::string store_value(const std::string& v, int node) {
        int odt = it.bufs[0].dtype;
        Cls vc = cls(node);
        switch (dtype_cls(odt)) {
            case CF16: return vc == CF16 ? v : "__float2half_rn(" + to_float(node, v) + ")";
            case CF32: {
                std::string f = to_float(node, v);
                return odt == DT_BF16 ? "__int_as_float(__float_as_int(" + f + ") & 0xFFFF0000)" : f;
            }
            case CINT: return vc == CBOOL ? "(" + v + " ? 1 : 0)" : "(int)(" + v + ")";
            default: return vc == CBOOL ? "(" + v + " ? 1u : 0u)" : "(unsigned)(" + v + ")";
        }
    }

    // ── kernel assembly ────────────────────────────────────────────────────────────────────────
    static const char* preamble() {
        return
            "#include <cuda_fp16.h>\n"
            // First statement of every kernel: nothing is read or written before the launch in front of this one has finished
            // (runtime.hpp, launch_kernel).  The next launch of the stream may place its blocks early only behind a grid of a few:
            // otherwise they take the places of this launch's own, or of one on the side stream, and idle there, and the
            // instruction is paid for by every block.  us with it in every kernel / in none / up to 32 blocks: sums over 56 for
            // 114688 outputs (14336 blocks) 18 / 12.4 / 12.4, column sums of 8192 x 4096 f16 30 / 15.6 / 15.6; symbolic f32 step at 17
            // rows 134 / 126 / 126, CNN step 82 / 77 / 77, f16 step at 1024 x 1024 155 / 148 / 148, f32 MLP step 24.8 / 26.3 / 25.2.
            "__device__ __forceinline__ void enter_() { if ((unsigned long long)gridDim.x * gridDim.y * gridDim.z <= 32u) asm volatile(\"griddepcontrol.launch_dependents;\"); asm volatile(\"griddepcontrol.wait;\" ::: \"memory\"); }\n"
            "__device__ __forceinline__ int clampi_(int i, int hi) { return i < 0 ? 0 : (i > hi ? hi : i); }\n"
            "__device__ __forceinline__ int idiv_(int a, int b) { return b == 0 ? 0 : a / b; }\n"
            "__device__ __forceinline__ int imod_(int a, int b) { return b == 0 ? 0 : a % b; }\n"
            "template <int BYTES> struct vec_t_;\n"
            "template <> struct vec_t_<16> { typedef uint4 type; };\n"
            "template <> struct vec_t_<8> { typedef uint2 type; };\n"
            "template <> struct vec_t_<4> { typedef unsigned type; };\n"
            "template <> struct vec_t_<2> { typedef unsigned short type; };\n"
            "template <class T, int V> __device__ __forceinline__ void ldv_(const T* p, T* out) {\n"
            "  typedef typename vec_t_<sizeof(T) * V>::type W;\n"
            "  W w = __ldg(reinterpret_cast<const W*>(p));\n"
            "  *reinterpret_cast<W*>(out) = w;\n"
            "}\n"
            "template <class T, int V> __device__ __forceinline__ void stv_(T* p, const T* in) {\n"
            "  typedef typename vec_t_<sizeof(T) * V>::type W;\n"
            "  *reinterpret_cast<W*>(p) = *reinterpret_cast<const W*>(in);\n"
            "}\n"
            // f16-class exp2 and reciprocal: one MUFU on the widened value, rounded back to f16.  The
            // f32 approximation is within 2 ulp (f32), far below the f16 rounding that follows.
            "__device__ __forceinline__ float ex2_h_(float x) { float r; asm(\"ex2.approx.ftz.f32 %0, %1;\" : \"=f\"(r) : \"f\"(x)); return r; }\n"
            "__device__ __forceinline__ float rcp_h_(float x) { float r; asm(\"rcp.approx.ftz.f32 %0, %1;\" : \"=f\"(r) : \"f\"(x)); return r; }\n"
            "#define DEF_H2MAP_(NAME, F) __device__ __forceinline__ __half2 NAME(__half2 x) { return __floats2half2_rn(F(__low2float(x)), F(__high2float(x))); }\n"
            "DEF_H2MAP_(h2_ex2_, ex2_h_)\n"
            "DEF_H2MAP_(h2_rcp_, rcp_h_)\n"
            "DEF_H2MAP_(h2_log2_, log2f)\n"
            "DEF_H2MAP_(h2_sqrt_, sqrtf)\n"
            "DEF_H2MAP_(h2_sin_, sinf)\n"
            "__device__ __forceinline__ __half2 h2_sel_(unsigned m, __half2 a, __half2 b) {\n"
            "  unsigned x = *reinterpret_cast<unsigned*>(&a), y = *reinterpret_cast<unsigned*>(&b), r = (x & m) | (y & ~m);\n"
            "  return *reinterpret_cast<__half2*>(&r);\n"
            "}\n"
            "__device__ __forceinline__ float op_add_f(float a, float b) { return a + b; }\n"
            "__device__ __forceinline__ float op_mul_f(float a, float b) { return a * b; }\n"
            "__device__ __forceinline__ float op_max_f(float a, float b) { return fmaxf(a, b); }\n"
            "__device__ __forceinline__ int op_add_i(int a, int b) { return a + b; }\n"
            "__device__ __forceinline__ int op_mul_i(int a, int b) { return a * b; }\n"
            "__device__ __forceinline__ int op_max_i(int a, int b) { return a > b ? a : b; }\n"
            // Combine the partial accumulators of the LANES threads that share one output.  RC layout:
            // the lanes of a group are consecutive threads; OC layout: they are TOUTS threads apart.
            // The combine order is fixed, so a kernel gives the same bits on every run.
            "#define DEF_GROUP_(NAME, T, OP) \\\n"
            "__device__ __forceinline__ T NAME(T v, int lane, int grp, float* sm) { \\\n"
            "  if (LANES == 1) return v; \\\n"
            "  if (RC_LAYOUT) { \\\n"
            "    _Pragma(\"unroll\") for (int o = (LANES < 32 ? LANES : 32) / 2; o > 0; o >>= 1) v = OP(v, __shfl_xor_sync(0xffffffffu, v, o)); \\\n"
            "    if (LANES > 32) { \\\n"
            "      T* s = reinterpret_cast<T*>(sm); \\\n"
            "      __syncthreads(); \\\n"
            "      if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v; \\\n"
            "      __syncthreads(); \\\n"
            "      const int w0 = grp * (LANES / 32); \\\n"
            "      v = s[w0]; \\\n"
            "      for (int w = 1; w < LANES / 32; w++) v = OP(v, s[w0 + w]); \\\n"
            "    } \\\n"
            "    return v; \\\n"
            "  } else { \\\n"
            "    T* s = reinterpret_cast<T*>(sm); \\\n"
            "    __syncthreads(); \\\n"
            "    s[lane * TOUTS + grp] = v; \\\n"
            "    __syncthreads(); \\\n"
            "    v = s[grp]; \\\n"
            "    for (int l = 1; l < LANES; l++) v = OP(v, s[l * TOUTS + grp]); \\\n"
            "    return v; \\\n"
            "  } \\\n"
            "}\n"
            "DEF_GROUP_(group_add_f, float, op_add_f)\n"
            "DEF_GROUP_(group_mul_f, float, op_mul_f)\n"
            "DEF_GROUP_(group_max_f, float, op_max_f)\n"
            "DEF_GROUP_(group_add_i, int, op_add_i)\n"
            "DEF_GROUP_(group_mul_i, int, op_mul_i)\n"
            "DEF_GROUP_(group_max_i, int, op_max_i)\n"
            // A reduction shared by nparts blocks.  Each leaves its partial in scratch memory and takes a ticket of
            // its output block; the one that takes the last ticket adds the parts up in a fixed order (whoever
            // it is, the same bits), puts the ticket word back to zero for the next launch and goes on to the
            // epilogue; the others are done (false).
            "#define DEF_JOIN_(NAME, T, OP, GROUP) \\\n"
            "__device__ __forceinline__ bool NAME(T& v, T ident, int lane, int grp, float* sm, unsigned* last, float* scratch, unsigned* tickets, int ob, int part, int nparts, int nob) { \\\n"
            "  T* sc = reinterpret_cast<T*>(scratch) + (long long)ob * TOUTS + grp; \\\n"
            "  const long long stride = (long long)nob * TOUTS; \\\n"
            "  if (lane == 0) sc[part * stride] = v; \\\n"
            "  __threadfence(); \\\n"
            "  __syncthreads(); \\\n"
            "  if (threadIdx.x == 0) { *last = atomicAdd(tickets + ob, 1u) == (unsigned)nparts - 1u; if (*last) tickets[ob] = 0u; } \\\n"
            "  __syncthreads(); \\\n"
            "  if (!*last) return false; \\\n"
            "  __threadfence(); \\\n"
            "  T w = ident; \\\n"
            "  for (int p = lane; p < nparts; p += LANES) w = OP(w, __ldcg(sc + p * stride)); \\\n"
            "  v = GROUP(w, lane, grp, sm); \\\n"
            "  return true; \\\n"
            "}\n";
    }
    // Combine the accumulators of the LANES threads that hold one row, one barrier each: every reduction of a row has a
    // shared-memory segment of its own, and each warp adds up the warps' values for itself.
    static const char* row_preamble() {
        return
            "template <int BYTES> __device__ __forceinline__ void fetch_(unsigned char* to, const void* from) {\n"
            "  const unsigned a = (unsigned)__cvta_generic_to_shared(to);\n"
            "  if (BYTES == 16) asm volatile(\"cp.async.cg.shared.global [%0], [%1], 16;\" :: \"r\"(a), \"l\"(from) : \"memory\");\n"
            "  else asm volatile(\"cp.async.ca.shared.global [%0], [%1], %2;\" :: \"r\"(a), \"l\"(from), \"n\"(BYTES == 16 ? 8 : BYTES) : \"memory\");\n"
            "}\n"
            "__device__ __forceinline__ void fetched_() { asm volatile(\"cp.async.wait_all;\" ::: \"memory\"); }\n"
            "template <class T, int V> __device__ __forceinline__ void take_(const unsigned char* from, T* out) {\n"
            "  typedef typename vec_t_<sizeof(T) * V>::type W;\n"
            "  *reinterpret_cast<W*>(out) = *reinterpret_cast<const W*>(from);\n"
            "}\n"
            "#define DEF_ROW_(NAME, T, OP) \\\n"
            "__device__ __forceinline__ T NAME(T v, float* sm) { \\\n"
            "  if (LANES == 1) return v; \\\n"
            "  _Pragma(\"unroll\") for (int o = 16; o > 0; o >>= 1) v = OP(v, __shfl_xor_sync(0xffffffffu, v, o)); \\\n"
            "  if (LANES > 32) { \\\n"
            "    T* s = reinterpret_cast<T*>(sm); \\\n"
            "    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v; \\\n"
            "    __syncthreads(); \\\n"
            "    v = s[threadIdx.x & (LANES / 32 - 1)]; \\\n"
            "    _Pragma(\"unroll\") for (int o = LANES / 64; o > 0; o >>= 1) v = OP(v, __shfl_xor_sync(0xffffffffu, v, o)); \\\n"
            "  } \\\n"
            "  return v; \\\n"
            "}\n"
            "DEF_ROW_(row_add_f, float, op_add_f)\n"
            "DEF_ROW_(row_mul_f, float, op_mul_f)\n"
            "DEF_ROW_(row_max_f, float, op_max_f)\n"
            "DEF_ROW_(row_add_i, int, op_add_i)\n"
            "DEF_ROW_(row_mul_i, int, op_mul_i)\n"
            "DEF_ROW_(row_max_i, int, op_max_i)\n";
    }
    static const char* join_preamble() {
        return
            "DEF_JOIN_(join_add_f, float, op_add_f, group_add_f)\n"
            "DEF_JOIN_(join_mul_f, float, op_mul_f, group_mul_f)\n"
            "DEF_JOIN_(join_max_f, float, op_max_f, group_max_f)\n"
            "DEF_JOIN_(join_add_i, int, op_add_i, group_add_i)\n"
            "DEF_JOIN_(join_mul_i, int, op_mul_i, group_mul_i)\n"
            "DEF_JOIN_(join_max_i, int, op_max_i, group_max_i)\n";
    }

    std::string signature(const std::string& name, bool with_scratch, int nthreads) {
        std::string s = "extern \"C\" __global__ void __launch_bounds__(" + std::to_string(nthreads) + ") " + name + "(";
        for (size_t b = 0; b < it.bufs.size(); b++) {
            s += (b ? ", " : "");
            s += (b ? "const " : "");
            s += buf_ctype(it.bufs[b].dtype);
            s += "* __restrict__ data" + std::to_string(b);
        }
        if (with_scratch) s += ", float* scratch, unsigned* tickets";
        if (has_sym) s += ", const int n0";
        if (with_scratch && has_sym) s += ", const int nsplit";
        return s + ")";
    }

    int64_t static_total() const {
        int64_t t = 1;
        for (int r : loop_ranges) if (!N(r).symbolic()) t *= N(r).arg;
        return t;
    }
    bool sym_output() const { for (int r : loop_ranges) if (N(r).symbolic()) return true; return false; }
    std::string total_expr() const {
        return sym_output() ? "((long long)n0 * " + std::to_string(static_total()) + ")" : std::to_string(static_total()) + "LL";
    }

    // r_i = (g / stride_i) % size_i for loop ranges [first, last), innermost last
    std::string decompose(const std::string& g, size_t first = 0, size_t last = (size_t)-1, const std::string& indent = "  ") {
        if (last == (size_t)-1) last = loop_ranges.size();
        std::string s;
        int64_t stride = 1;
        for (int k = (int)last - 1; k >= (int)first; k--) {
            int r = loop_ranges[k];
            std::string rn = "r" + std::to_string(N(r).aux);
            std::string e = stride == 1 ? g : "(" + g + " / " + std::to_string(stride) + ")";
            if (k == (int)first || N(r).symbolic()) s += indent + "const int " + rn + " = (int)" + e + ";\n";
            else s += indent + "const int " + rn + " = (int)(" + e + " % " + std::to_string(N(r).arg) + ");\n";
            if (!N(r).symbolic()) stride *= N(r).arg;
        }
        return s;
    }

    void reset_emit() { top = Block(); prelude = Block(); cur_top = nullptr; loop.clear(); memo.clear(); vec_load.clear(); vec_range = -1; reduce_vec = 1; }

    // vector width the elementwise path may use, and the loads it can preload as vectors
    int pick_vector(std::vector<int>& vloads) {
        if (opts.vector_width == 1 || loop_ranges.empty() || opts.debug_bounds) return 1;
        int rv = loop_ranges.back();
        if (N(rv).symbolic()) return 1;
        bool all16 = dt_storage_bytes(it.bufs[0].dtype) == 2;
        std::vector<int> idx_nodes;
        for (int i = 0; i < n; i++) if (N(i).op == OP_INDEX && i != dst && is_live(i)) idx_nodes.push_back(i);
        for (int i : idx_nodes) if (dt_storage_bytes(it.bufs[(int)N(N(i).src[0]).arg].dtype) != 2) { all16 = false; }
        int V = opts.vector_width > 1 ? opts.vector_width : (all16 ? 8 : 4);
        if (!all16 && V > 4) V = 4;            // one access is at most 128 bits
        if (V != 4 && V != 8 && V != 2) V = all16 ? 8 : 4;
        if (N(rv).arg % V != 0) return 1;
        vloads.clear();
        for (int i : idx_nodes) {
            int p = (int)N(N(i).src[0]).arg;
            Lin f = flat_index(i);
            bool ok; int64_t c = lin_coef(f, rv, ok);
            if (!ok) return 1;                 // the unrolled variable is buried in a div/mod
            if (c == 0) continue;              // broadcast along the vector
            if (c != 1) return 1;
            if (!in_bounds(f, p)) return 1;
            if (f.c % V != 0) return 1;
            for (auto& t : f.t) {
                const Atom& a = atoms[t.first];
                if (a.kind == Atom::RANGE && a.node == rv) continue;
                if (t.second % V != 0) return 1;
            }
            vloads.push_back(i);
        }
        return V;
    }
    std::vector<bool> live_;
    bool is_live(int i) {
        if (live_.empty()) {
            live_.assign(n, false);
            std::function<void(int)> mark = [&](int k) { if (live_[k]) return; live_[k] = true; for (int s : N(k).src) mark(s); };
            mark(body);
        }
        return live_[i];
    }

    // The body once per combination of the enumerated output ranges, as the cases of a switch; inside a case they are constants.
    bool emit_cases(std::ostringstream& k, const std::string& store_to) {
        std::string sel = "0";
        int64_t cases = 1;
        for (int r : enum_out) { sel = "(" + sel + " * " + std::to_string(N(r).arg) + " + r" + std::to_string(N(r).aux) + ")"; cases *= N(r).arg; }
        k << "  switch (" << sel << ") {\n";
        for (int64_t cs = 0; cs < cases; cs++) {
            int64_t rem = cs;
            for (int e = (int)enum_out.size() - 1; e >= 0; e--) { fix_range(enum_out[e], rem % N(enum_out[e]).arg); rem /= N(enum_out[e]).arg; }
            top = Block(); loop.clear(); memo.clear();
            std::string v = val(body, -1);
            if (!err.empty()) return false;
            k << "  case " << cs << ": {\n" << top.code;
            k << store_to << store_value(v, body) << ";\n  } break;\n";
        }
        for (int r : enum_out) unfix_range(r);
        k << "  }\n";
        return true;
    }

    bool build_elementwise(Rendered& out) {
        std::vector<int> vloads;
        int V = pick_vector(vloads);
        int T = opts.block_threads > 0 ? opts.block_threads : 256;
        reset_emit();
        std::ostringstream k;
        k << "#define LANES 1\n#define TOUTS 1\n#define RC_LAYOUT 1\n";
        k << preamble();
        std::string name = "ew_fused";
        k << signature(name, false, T) << " {\n  enter_();\n";
        k << "  const long long g = (long long)blockIdx.x * " << T << " + threadIdx.x;\n";
        if (V == 1) {
            k << "  if (g >= " << total_expr() << ") return;\n";
            k << decompose("g");
            if (!enum_out.empty()) {
                if (!emit_cases(k, "  data0[g] = ")) return false;
            } else {
                std::string v = val(body, -1);
                if (!err.empty()) return false;
                k << top.code;
                k << "  data0[g] = " << store_value(v, body) << ";\n";
            }
        } else {
            int rv = loop_ranges.back();
            h2 = opts.vector_width >= 0 && h2_eligible(V);
            const int U = h2 ? V / 2 : V;                  // iterations of the unrolled loop
            k << "  const long long base = g * " << V << ";\n";
            k << "  if (base >= " << total_expr() << ") return;\n";
            k << decompose("base");
            // preload the unit-stride operands with one wide access each
            vec_range = -1;
            int vi = 0;
            cur_top = &prelude;
            for (int i : vloads) {
                int p = (int)N(N(i).src[0]).arg;
                Lin f = flat_index(i);
                std::string arr = "v" + std::to_string(vi++);
                std::string bt = buf_ctype(it.bufs[p].dtype), VS = std::to_string(V);
                std::string idx = render(f, -1);
                if (h2) {
                    stmt(-1, "__half2 " + arr + "_raw[" + std::to_string(U) + "];");
                    stmt(-1, "ldv_<__half2, " + std::to_string(U) + ">(reinterpret_cast<const __half2*>(data" + std::to_string(p) + " + " + idx + "), " + arr + "_raw);");
                    vec_load[i] = arr + "_raw";
                    continue;
                }
                stmt(-1, bt + " " + arr + "_raw[" + VS + "];");
                stmt(-1, "ldv_<" + bt + ", " + VS + ">(data" + std::to_string(p) + " + " + idx + ", " + arr + "_raw);");
                // convert to the compute class of the INDEX node
                Cls bc = dtype_cls(it.bufs[p].dtype), want = cls(i);
                if (dtype_cls(N(i).dtype) == CBOOL) {
                    stmt(-1, "bool " + arr + "[" + VS + "];");
                    stmt(-1, "_Pragma(\"unroll\") for (int u = 0; u < " + VS + "; u++) " + arr + "[u] = " + arr + "_raw[u] != 0u;");
                    vec_load[i] = arr;
                } else if (bc == CF16 && want == CF32) {
                    stmt(-1, "float " + arr + "[" + VS + "];");
                    stmt(-1, "_Pragma(\"unroll\") for (int u = 0; u < " + VS + "; u++) " + arr + "[u] = __half2float(" + arr + "_raw[u]);");
                    vec_load[i] = arr;
                } else {
                    vec_load[i] = arr + "_raw";
                }
            }
            cur_top = nullptr;
            vec_range = rv;
            std::string v = h2 ? val_h2(body) : val(body, -1);
            if (!err.empty()) return false;
            k << prelude.code;
            const std::string ot = h2 ? "__half2" : buf_ctype(it.bufs[0].dtype);
            k << "  " << ot << " outv[" << U << "];\n";
            k << "  _Pragma(\"unroll\") for (int u = 0; u < " << U << "; u++) {\n";
            k << top.code;
            k << "    outv[u] = " << (h2 ? v : store_value(v, body)) << ";\n";
            k << "  }\n";
            if (h2) k << "  stv_<__half2, " << U << ">(reinterpret_cast<__half2*>(data0 + base), outv);\n";
            else k << "  stv_<" << ot << ", " << V << ">(data0 + base, outv);\n";
        }
        k << "}\n";
        out.klass = KC_ELEMENTWISE;
        out.source = k.str();
        out.vector_width = V;
        out.main.entry = name;
        out.main.block = T;
        out.main.outputs_per_block = (int64_t)T * V;
        out.main.static_outputs = static_total();
        out.main.sym_trailing = sym_output() ? static_total() : 0;
        out.uses_sym = has_sym;
        out.note = "elementwise V=" + std::to_string(V) + (h2 ? " paired f16" : "");
        if (V == 1 && !enum_out.empty()) out.note += " switch over " + std::to_string(enum_out.size()) + " output ranges";
        return true;
    }

    // flattened size of a REDUCE's ranges; 0 if symbolic
    int64_t reduce_total(int r) const {
        int64_t t = 1;
        for (size_t s = 1; s < N(r).src.size(); s++) {
            int rn = N(r).src[s];
            if (N(rn).op != OP_RANGE) continue;
            if (N(rn).symbolic()) return 0;
            t *= N(rn).arg;
        }
        return t;
    }

    // smallest element a load inside this REDUCE reads
    int reduce_load_bytes(int red) {
        int bytes = 4;
        for (int i = 0; i < n; i++)
            if (N(i).op == OP_INDEX && i != dst && is_live(i) && depends_on_reduce(i, red) && N(N(i).src[0]).op == OP_PARAM) bytes = std::min(bytes, dt_storage_bytes(it.bufs[(int)N(N(i).src[0]).arg].dtype));
        return bytes;
    }

    void choose_layout(int64_t total, int64_t rtot_max) {
        // votes: bytes of loads that are unit-stride along the innermost reduce range (RC) against
        // loads unit-stride along the innermost output range (OC)
        int64_t rc = 0, oc = 0;
        int oc_min_bytes = 4;
        int out_inner = loop_ranges.empty() ? -1 : loop_ranges.back();
        for (int r : reduces) {
            int red_inner = -1;
            for (size_t s = 1; s < N(r).src.size(); s++) if (N(N(r).src[s]).op == OP_RANGE) red_inner = N(r).src[s];
            if (red_inner < 0) continue;
            for (int i = 0; i < n; i++) {
                if (N(i).op != OP_INDEX || i == dst || !is_live(i) || !dep[i][range_slot[red_inner]]) continue;
                Lin f = flat_index(i);
                bool ok1, ok2 = false;
                int64_t c1 = lin_coef(f, red_inner, ok1);
                int64_t c2 = out_inner >= 0 ? lin_coef(f, out_inner, ok2) : 0;
                int bytes = dt_storage_bytes(it.bufs[(int)N(N(i).src[0]).arg].dtype);
                if (ok1 && std::llabs(c1) == 1) rc += bytes;
                else if (ok2 && std::llabs(c2) == 1) { oc += bytes; oc_min_bytes = std::min(oc_min_bytes, bytes); }
            }
        }
        threads = opts.block_threads > 0 ? opts.block_threads : 256;
        const int64_t want_threads = 148LL * 1024;     // enough to fill the machine
        if (oc > 0) {
            rc_layout = false;
            int L = 1;
            if (opts.reduce_lanes > 0) L = opts.reduce_lanes;
            else {
                while (L < 32 && total * L < want_threads && rtot_max / (L * 2) >= 16) L *= 2;
                // the threads that share a row cover TOUTS adjacent outputs: keep that run at least one
                // 32-byte sector wide, or every sector fetched is only partly used (f16: 16 outputs)
                const int min_touts = std::max(1, 32 / std::max(1, oc_min_bytes));
                while (L > 1 && threads / L < min_touts) L /= 2;
            }
            lanes = L;
        } else {
            rc_layout = true;
            int L;
            if (opts.reduce_lanes > 0) L = opts.reduce_lanes;
            else if (rtot_max == 0) L = 32;          // symbolic bound
            else if (rtot_max <= 16) L = 1;
            else if (rtot_max < 1024) { L = 32; while (L > rtot_max) L /= 2; }
            else L = threads;
            if (opts.reduce_lanes == 0 && L < threads && total * L < want_threads / 4 && rtot_max >= 64) {
                while (L < threads && total * L < want_threads / 4 && rtot_max / (L * 2) >= 4) L *= 2;
            }
            lanes = L;
        }
        if (!enum_reduce.empty() && opts.reduce_lanes == 0) lanes = 1;      // value-by-value loops are per thread
        if (lanes > threads) lanes = threads;
        touts = threads / lanes;
    }

    // `split`: parts per output, 0 = none, -1 = the kernel's nsplit argument.  `nob`: output blocks.  `wide`: elements a lane
    // may take at once.
    std::string reduce_macros(int split = 0, int64_t nob = 0, int wide = 8) {
        std::ostringstream m;
        m << "#define LANES " << lanes << "\n#define TOUTS " << touts << "\n#define RC_LAYOUT " << (rc_layout ? 1 : 0) << "\n";
        if (split) {
            // each of an output's blocks owns a contiguous chunk of the flattened reduce space, a multiple of `wide`
            // elements for every lane so that wide loads stay aligned
            const std::string unit = "(" + std::to_string(wide) + " * LANES)";
            m << "#define SPLIT " << (split < 0 ? std::string("nsplit") : std::to_string(split)) << "\n#define NOB " << nob << "\n";
            m << "#define RED_CHUNK(n) ((((n) + SPLIT - 1) / SPLIT + " << unit << " - 1) / " << unit << " * " << unit << ")\n";
            m << "#define RED_LO(n) ((int)min((long long)part * RED_CHUNK(n), (long long)(n)))\n";
            m << "#define RED_BEGIN(n) (RED_LO(n) + lane)\n#define RED_BEGIN_V(n, v) (RED_LO(n) + lane * (v))\n";
            m << "#define RED_END(n) ((int)min((long long)(part + 1) * RED_CHUNK(n), (long long)(n)))\n#define RED_STEP LANES\n";
        } else {
            m << "#define RED_BEGIN(n) lane\n#define RED_BEGIN_V(n, v) (lane * (v))\n#define RED_END(n) (n)\n#define RED_STEP LANES\n";
        }
        return m.str();
    }

    // The same stage when the row sits in registers.
    bool build_row_stage(int k, int threads_, std::string& decl, std::string& code, std::string& result_var, bool has_inner) {
        threads = threads_; lanes = threads_; touts = 1; rc_layout = true;
        reset_emit();
        dp = "s" + std::to_string(k) + "_data";
        std::ostringstream c;
        const std::string bt = buf_ctype(it.bufs[0].dtype);
        result_var = "stage" + std::to_string(k);
        if (!has_inner) decl = "  " + bt + " " + result_var + ";\n";
        c << "  {   // stage " << k << "\n  const int r" << N(loop_ranges[0]).aux << " = row; (void)r" << N(loop_ranges[0]).aux << ";\n";
        cur_top = &prelude;
        for (int r : reduces) { val(r, -1); if (!err.empty()) return false; }
        cur_top = nullptr;
        const std::string v = val(body, -1);
        if (!err.empty()) return false;
        c << prelude.code;
        if (!has_inner) {
            c << top.code << "  " << result_var << " = " << store_value(v, body) << ";\n  if (lane == 0) " << dp << "0[row] = " << result_var << ";\n";
        } else {
            const int w = loop_ranges[1];
            const std::string V = std::to_string(row_vec), at = dp + "0 + ((long long)row * " + std::to_string(row_len) + "LL + cb)";
            c << "  " << bt << " outv[" << row_chunks * row_vec << "];\n" << row_open("r" + std::to_string(N(w).aux), row_loads_memory(body, w)) << top.code;
            c << "    outv[u] = " << store_value(v, body) << ";\n  }\n";
            if (row_shifted) {
                c << "    if (cb < 0 || cb + " << V << " > " << row_len << ") {\n      _Pragma(\"unroll\") for (int v = 0; v < " << V << "; v++) if ((unsigned)(cb + v) < " << row_len << "u) (" << at << ")[v] = outv[c * " << V << " + v];\n    } else\n";
            } else if (!row_exact()) c << "    if (live)\n";
            if (row_vec > 1) c << "    stv_<" << bt << ", " << V << ">(" << at << ", outv + c * " << V << ");\n  }\n";
            else c << "    *(" << at << ") = outv[c];\n  }\n";
        }
        c << "  }\n";
        code = c.str();
        return true;
    }

    // One stage of a row chain.  Requirements: static ranges, the first loop range is the row, every
    // REDUCE is invariant along the other loop ranges (they are swept after the reductions).  Emits
    //   <decl>  : declaration of the stage's per-row result (when the stage has no inner ranges)
    //   <code>  : a braced block computing it for row `row`
    bool build_chain_stage(int k, int threads_, std::string& decl, std::string& code, std::string& result_var, int64_t& rows, bool& has_inner) {
        if (!analyse()) return false;
        if (has_sym || loop_ranges.empty()) return fail("chain: symbolic or scalar kernel");
        rows = N(loop_ranges[0]).arg;
        for (size_t r = 1; r < loop_ranges.size(); r++)
            for (int red : reduces) if (dep[red][range_slot[loop_ranges[r]]]) return fail("chain: a reduction depends on an inner output range");
        // every load must be unit-stride (or constant) along the innermost range it sweeps inside the row,
        // otherwise one block per row would stride through memory (a column sum is not a row chain)
        for (int i = 0; i < n; i++) {
            if (N(i).op != OP_INDEX || i == dst || !is_live(i)) continue;
            int innermost = -1;
            for (int r : all_ranges) if (r != loop_ranges[0] && dep[i][range_slot[r]]) innermost = std::max(innermost, r);
            if (innermost < 0) continue;
            bool ok; int64_t c = lin_coef(flat_index(i), innermost, ok);
            if (!ok || std::llabs(c) > 1) return fail("chain: strided access inside the row");
        }
        has_inner = loop_ranges.size() > 1;
        if (row_len > 0) return build_row_stage(k, threads_, decl, code, result_var, has_inner);
        int64_t inner = 1;
        for (size_t r = 1; r < loop_ranges.size(); r++) inner *= N(loop_ranges[r]).arg;
        threads = threads_; lanes = threads; touts = 1; rc_layout = true;
        reset_emit();
        reduce_combine_mode = "group";
        unroll_short_loops = true;
        // 4-element chunks per lane with explicit 128-bit loads and stores where a row allows it
        chain_vec = 4;
        dp = "s" + std::to_string(k) + "_data";
        std::ostringstream c;
        std::string bt = buf_ctype(it.bufs[0].dtype);
        result_var = "stage" + std::to_string(k);
        if (!has_inner) decl = "  " + bt + " " + result_var + ";\n";
        c << "  {   // stage " << k << "\n";
        c << "  const int r" << N(loop_ranges[0]).aux << " = row;\n";
        cur_top = &prelude;
        for (int r : reduces) { val(r, -1); if (!err.empty()) return false; }
        cur_top = nullptr;
        // the last stage writes the row in chunks of chain_vec outputs per lane: wide loads of its
        // unit-stride operands, one wide store
        const Cls oc = dtype_cls(it.bufs[0].dtype);
        const bool chunk_sweep = has_inner && chain_vec > 1 && inner <= (int64_t)threads * 32 && inner % ((int64_t)threads * chain_vec) == 0 &&
                                 N(loop_ranges.back()).arg % chain_vec == 0 && (oc == CF32 || oc == CF16) && it.bufs[0].dtype != DT_BF16;
        std::string wide;
        if (chunk_sweep) wide = chain_wide_loads(body, loop_ranges.back(), -1);
        std::string v = val(body, -1);
        if (!err.empty()) return false;
        c << prelude.code;
        if (has_inner) {
            if (chunk_sweep) {
                c << "  _Pragma(\"unroll\") for (int gb = threadIdx.x * " << chain_vec << "; gb < " << inner << "; gb += " << threads * chain_vec << ") {\n";
                c << "    " << bt << " outv[" << chain_vec << "];\n";
                // the loads are written with the chunk's first index; the per-element scope below shadows it
                c << "    const int gi = gb; (void)gi;\n" << decompose("gi", 1, loop_ranges.size(), "    ") << wide;
                c << "  _Pragma(\"unroll\") for (int u = 0; u < " << chain_vec << "; u++) { const int gi = gb + u;\n";
            } else {
                c << (inner <= (int64_t)threads * 32 ? "  _Pragma(\"unroll\")\n" : "");
                c << "  for (int gi = threadIdx.x; gi < " << inner << "; gi += " << threads << ") {\n";
            }
            c << decompose("gi", 1, loop_ranges.size(), "    ");
            c << top.code;
            if (chunk_sweep) {
                c << "    outv[u] = " << store_value(v, body) << ";\n  }\n";
                c << "    stv_<" << bt << ", " << chain_vec << ">(" << dp << "0 + ((long long)row * " << inner << "LL + gb), outv);\n";
            } else c << "    " << dp << "0[(long long)row * " << inner << "LL + gi] = " << store_value(v, body) << ";\n";
            c << "  }\n";
        } else {
            c << top.code;
            c << "  " << result_var << " = " << store_value(v, body) << ";\n";
            c << "  if (threadIdx.x == 0) " << dp << "0[row] = " << result_var << ";\n";
        }
        c << "  }\n";
        code = c.str();
        return true;
    }

    // Every REDUCE is invariant along the trailing `ninv` output ranges (a row statistic consumed by
    // an elementwise expression over the row, the shape epilogue fusion produces for softmax-like
    // graphs, schedule/schedule.go:197-233).  The reference re-runs the reduction for every output
    // element; here one block owns one outer index, all threads cooperate on each reduction once,
    // then sweep the invariant ranges.
    bool build_rowbcast(Rendered& out, size_t ninv, int64_t inner) {
        threads = opts.block_threads > 0 ? opts.block_threads : 256;
        lanes = threads; touts = 1; rc_layout = true;
        size_t nouter = loop_ranges.size() - ninv;
        int64_t outer = 1; bool osym = false;
        for (size_t k = 0; k < nouter; k++) { if (N(loop_ranges[k]).symbolic()) osym = true; else outer *= N(loop_ranges[k]).arg; }
        reset_emit();
        reduce_combine_mode = "group";
        std::ostringstream k;
        k << reduce_macros() << preamble();
        std::string name = "reduce_rowbcast";
        row_broadcast = true;
        k << signature(name, false, threads) << " {\n  enter_();\n";
        k << "  __shared__ float red_smem[" << std::max(threads / 32, 1) << "];\n";
        k << "  const int lane = threadIdx.x, grp = 0;\n";
        k << "  const long long go = blockIdx.x;\n";
        k << decompose("go", 0, nouter);
        cur_top = &prelude;
        for (int r : reduces) { val(r, -1); if (!err.empty()) return false; }
        cur_top = nullptr;
        std::string v = val(body, -1);
        if (!err.empty()) return false;
        k << prelude.code;
        k << "  for (int gi = threadIdx.x; gi < " << inner << "; gi += " << threads << ") {\n";
        k << decompose("gi", nouter, loop_ranges.size(), "    ");
        k << top.code;
        k << "    data0[go * " << inner << "LL + gi] = " << store_value(v, body) << ";\n";
        k << "  }\n}\n";
        out.klass = KC_REDUCE;
        out.source = k.str();
        out.main.entry = name;
        out.main.block = threads;
        out.main.outputs_per_block = 1;
        out.main.static_outputs = outer;
        out.main.sym_trailing = osym ? outer : 0;
        out.uses_sym = has_sym;
        out.note = "reduce row-broadcast inner=" + std::to_string(inner) + " lanes=" + std::to_string(lanes);
        return true;
    }

    // value of an affine form for given loop variables; `known` is cleared where it hangs on something else
    int64_t lin_at(const Lin& l, const std::map<int, int64_t>& at, bool& known) const {
        int64_t v = l.c;
        for (auto& p : l.t) {
            const Atom& a = atoms[p.first];
            if (a.kind == Atom::RANGE) { auto f = at.find(a.node); v += p.second * (f == at.end() ? 0 : f->second); }
            else if (a.kind == Atom::OPAQUE) known = false;
            else { const int64_t x = lin_at(a.inner, at, known); v += p.second * (a.kind == Atom::DIV ? x / a.d : x % a.d); }
        }
        return v;
    }
    // 128-byte lines that a warp touches per output when neighbouring threads take neighbouring values of `order`'s last range:
    // the loads `refs` and the store; averaged over a few warps.  < 0: not known.
    double lines_touched(const std::vector<int>& order, const std::vector<std::pair<Lin, int>>& refs) {
        const int64_t total = static_total();
        double sum = 0;
        const int64_t starts[4] = {0, total / 4 / 32 * 32, total / 2 / 32 * 32, total * 3 / 4 / 32 * 32};
        for (int64_t g0 : starts) {
            std::vector<std::set<int64_t>> seen(refs.size() + 1);
            for (int64_t g = g0; g < g0 + 32 && g < total; g++) {
                std::map<int, int64_t> at;
                int64_t rem = g;
                for (size_t k = order.size(); k-- > 0;) { at[order[k]] = rem % N(order[k]).arg; rem /= N(order[k]).arg; }
                bool known = true;
                for (size_t r = 0; r < refs.size(); r++) seen[r].insert(lin_at(refs[r].first, at, known) * refs[r].second >> 7);
                int64_t o = 0;
                for (int r : loop_ranges) o = o * N(r).arg + at[r];
                seen.back().insert(o * dt_storage_bytes(it.bufs[0].dtype) >> 7);
                if (!known) return -1;
            }
            for (auto& l : seen) sum += (double)l.size();
        }
        return sum / 4;
    }
    // Which range neighbouring threads should differ in when every thread works out one output by itself: the last one, unless
    // another more than halves the lines touched.  A convolution with its channels last reads 16 channels' weights 288
    // bytes apart in every warp; with the positions last they are one address and the image is contiguous: alone, 6 us of
    // timing events included, 32 x 196 x 16 outputs of 72 taps 12.4 -> 9.2 us, 128 x 576 x 24 of 108 taps 197 -> 65.
    std::vector<int> thread_order() {
        std::vector<int> best = loop_ranges;
        std::vector<std::pair<Lin, int>> refs;
        loads_seen = &refs;
        val(body, -1);
        loads_seen = nullptr;
        reset_emit();
        const double as_is = lines_touched(loop_ranges, refs);
        double least = as_is / 2;
        if (as_is < 0) return best;
        for (size_t k = 0; k + 1 < loop_ranges.size(); k++) {
            if (N(loop_ranges[k]).arg < 16) continue;
            std::vector<int> o = loop_ranges;
            o.erase(o.begin() + k);
            o.push_back(loop_ranges[k]);
            const double c = lines_touched(o, refs);
            if (c >= 0 && c < least) { least = c; best = o; }
        }
        return best;
    }

    // The enumerated outputs of a long reduction side by side: the innermost of the enumerated ranges (the 3 x 3 taps of a
    // convolution's weight gradient) become accumulators of one thread, the others stay a switch.  As a block per output
    // such a kernel reads the gradient once per tap and works out the same indexes (divisions by the image's extents, borders)
    // for every term of every output, which is what bounded it.  Alone, 6 us of timing events included: 16 x 8 x 3 x 3
    // outputs of 6272 terms 26.6 -> 11.3 us, 24 x 12 x 3 x 3 of 73728 218 -> 80, 8 x 1 x 3 x 3 of 25088 13.3 -> 10.2, 12 x 1 x 3 x 3 of
    // 294912 53 -> 31.
    bool build_side_by_side(Rendered& out, int64_t rmax, bool& taken) {
        taken = false;
        size_t nin = 0; int64_t ninner = 1;
        while (nin < loop_ranges.size()) {
            const int r = loop_ranges[loop_ranges.size() - 1 - nin];
            if (std::find(enum_out.begin(), enum_out.end(), r) == enum_out.end() || ninner * N(r).arg > 16) break;
            ninner *= N(r).arg; nin++;
        }
        if (nin == 0 || ninner < 4 || rmax < 1024) return true;
        const std::vector<int> inner(loop_ranges.end() - nin, loop_ranges.end());
        std::vector<int> outer;
        for (int r : enum_out) if (std::find(inner.begin(), inner.end(), r) == inner.end()) outer.push_back(r);
        auto fix_all = [&](const std::vector<int>& rs, int64_t v) { for (size_t e = rs.size(); e-- > 0;) { fix_range(rs[e], v % N(rs[e]).arg); v /= N(rs[e]).arg; } };
        int64_t cases = 1;
        for (int r : outer) cases *= N(r).arg;
        // Many groups: a block of up to 1024 lanes each.  Few: parts of one trip a lane in up to 16 blocks a group, from
        // three trips on wider blocks and then more of them while the SMs have room, as a block's trips are one chain of
        // latencies; one block where a lane of it has a trip or two, as the ticket and the second pass cost as much.  us a launch in a row of sixteen, groups x
        // terms, a block per output (no such form) | parts of four trips a lane | this: 4 x 1200 4.0 | 6.1 | 4.1, 6 x 2000 5.8 | 6.9 | 4.0,
        // 8 x 2048 5.4 | 5.8 | 3.8, 8 x 6272 13.5 | 6.9 | 4.9, 8 x 25088 20 | 8.6 | 7.5, 4 x 73728 18.5 | 9.8 | 9.8, 64 x 18432 62 | 18 | 14;
        // in one block 64 x 1152 4.8 | 5.8 | 4.1, 4 x 1024 3.8 | 3.9 | 3.4.
        const int64_t groups = static_total() / ninner;
        int L = 256, parts = 1;
        if (groups >= 74) { while (L < 1024 && groups * L < 148 * 1024 && rmax / (L * 2) >= 4) L *= 2; }
        else if (rmax <= (groups >= 32 ? 1280 : 1024)) L = 1024;
        else {
            parts = (int)std::min<int64_t>({(rmax + L - 1) / L, 512 / groups, 16});
            while (groups * parts * L * 2 <= 148 * 1024 && rmax > 3ll * L * parts) { if (L < 1024) L *= 2; else parts *= 2; }
        }
        if (groups > kMaxTickets && parts > 1) parts = 1;
        rc_layout = true; lanes = threads = L; touts = 1;

        const int red = reduces[0], rop = (int)N(red).aux;
        const Cls c0 = dtype_cls(N(red).dtype);
        const bool isf = c0 == CF32 || c0 == CF16;
        const Cls acc_c = isf ? CF32 : c0;
        const std::string tag = std::string(rop_tag(rop)) + "_" + (isf ? "f" : "i"), at = isf ? "float" : cls_ctype(acc_c);
        reset_emit();
        reduce_combine_mode.clear();
        std::string text;
        for (int64_t cs = 0; cs < cases && side.ok; cs++) {
            fix_all(outer, cs);
            std::string decl, head, body_text, group, finish;
            for (int64_t in = 0; in < ninner && side.ok; in++) {
                fix_all(inner, in);
                top = Block(); loop.clear(); memo.clear();
                side = SideBySide(); side.on = true; side.tag = "_" + std::to_string(in);
                const std::string v = val(body, -1);
                if (!err.empty() || side.reds != 1) side.ok = false;
                const std::string num = std::to_string(in);
                decl += side.decl; head = side.head; body_text += side.body;
                group += "  _Pragma(\"unroll\") for (int o = 16; o > 0; o >>= 1) " + side.acc + " = op_" + tag + "(" + side.acc + ", __shfl_xor_sync(0xffffffffu, " + side.acc + ", o));\n" +
                         "  if ((threadIdx.x & 31) == 0) sums[" + num + " * (LANES / 32) + (threadIdx.x >> 5)] = " + side.acc + ";\n";
                finish += "  if (lane == " + num + ") {\n  const " + at + " " + side.acc + " = mine;\n" + top.code + "  data0[g * " + std::to_string(ninner) + " + " + num + "] = " + store_value(v, body) + ";\n  }\n";
            }
            // the warps' sums together, added in order by one thread an output
            text += "  case " + std::to_string(cs) + ": {\n" + decl + head + body_text + "  }\n" + group + "  __syncthreads();\n";
            text += "  " + at + " mine = " + identity(rop, acc_c) + ";\n  if (lane < " + std::to_string(ninner) + ") { mine = sums[lane * (LANES / 32)]; for (int w = 1; w < LANES / 32; w++) mine = op_" + tag + "(mine, sums[lane * (LANES / 32) + w]); }\n";
            if (parts > 1) {
                const std::string cell = "NOB + ob) * " + std::to_string(ninner) + " + lane";
                text += "  " + at + "* const sc = reinterpret_cast<" + at + "*>(scratch);\n  if (lane < " + std::to_string(ninner) + ") { sc[((long long)part * " + cell + "] = mine; __threadfence(); }\n  __syncthreads();\n";
                text += "  if (threadIdx.x == 0) { split_last = atomicAdd(tickets + ob, 1u) == (unsigned)SPLIT - 1u; if (split_last) tickets[ob] = 0u; }\n";
                text += "  __syncthreads();\n  if (!split_last) return;\n  __threadfence();\n";
                text += "  if (lane < " + std::to_string(ninner) + ") { mine = " + identity(rop, acc_c) + "; _Pragma(\"unroll 8\") for (int p = 0; p < SPLIT; p++) mine = op_" + tag + "(mine, __ldcg(sc + ((long long)p * " + cell + ")); }\n";
            }
            text += finish + "  } break;\n";
        }
        for (int r : enum_out) unfix_range(r);
        const bool ok = side.ok && err.empty();
        side = SideBySide();
        if (!ok) return err.empty();
        std::ostringstream k;
        k << reduce_macros(parts > 1 ? parts : 0, groups, 1) << preamble();
        k << signature("reduce_fused", parts > 1, threads) << " {\n  enter_();\n";
        k << "  __shared__ " << at << " sums[" << ninner * (threads / 32) << "];\n  const int lane = threadIdx.x;\n";
        if (parts > 1) k << "  __shared__ unsigned split_last;\n  const int ob = blockIdx.x / SPLIT, part = blockIdx.x % SPLIT;\n  const long long g = ob;\n";
        else k << "  const long long g = blockIdx.x;\n";
        k << decompose("g", 0, loop_ranges.size() - nin);
        std::string sel = "0";
        for (int r : outer) sel = "(" + sel + " * " + std::to_string(N(r).arg) + " + r" + std::to_string(N(r).aux) + ")";
        k << "  switch (" << sel << ") {\n" << text << "  }\n}\n";
        out.klass = parts > 1 ? KC_REDUCE_SPLIT : KC_REDUCE;
        out.source = k.str();
        out.main.entry = "reduce_fused";
        out.main.block = threads;
        out.main.outputs_per_block = 1;
        out.main.static_outputs = groups;
        if (parts > 1) { out.split = parts; out.out_blocks = groups; out.part_elems = groups * ninner; out.split_lanes = lanes; }
        out.note = "reduce RC lanes=" + std::to_string(lanes) + " " + std::to_string(ninner) + " outputs side by side";
        if (parts > 1) out.note += " split reduce parts=" + std::to_string(parts);
        if (!outer.empty()) out.note += " switch over " + std::to_string(outer.size()) + " output ranges";
        taken = true;
        return true;
    }

    bool build_reduce(Rendered& out) {
        if (opts.reduce_lanes == 0 && opts.split <= 1 && !opts.sym_split && enum_out.empty() && enum_reduce.empty()) {
            size_t ninv = 0; int64_t inner = 1;
            for (int k = (int)loop_ranges.size() - 1; k >= 0; k--) {
                int r = loop_ranges[k];
                if (N(r).symbolic()) break;
                bool used = false;
                for (int red : reduces) if (dep[red][range_slot[r]]) used = true;
                if (used) break;
                ninv++; inner *= N(r).arg;
            }
            if (ninv > 0 && inner >= 64) return build_rowbcast(out, ninv, inner);
        }
        int64_t total = static_total();
        int64_t rmax = 0; bool rsym = false;
        for (int r : reduces) { int64_t t = reduce_total(r); if (t == 0) rsym = true; rmax = std::max(rmax, t); }
        if (!enum_out.empty() && enum_reduce.empty() && reduces.size() == 1 && !rsym && !sym_output() && opts.split <= 1 && opts.reduce_lanes == 0 && opts.block_threads == 0) {
            bool taken = false;
            if (!build_side_by_side(out, rmax, taken)) return false;
            if (taken) return true;
        }
        const bool dyn = opts.sym_split;         // the form of a REDUCE over the bound batch whose parts are counted at launch
        if (dyn && !(rsym && reduces.size() == 1 && !sym_output())) return fail("codegen: no split over the bound batch");
        if (rsym) rmax = dyn ? (int64_t)1 << 20 : 0;
        int64_t est_total = sym_output() ? total * (opts.sym_hint > 0 ? opts.sym_hint : 1024) : total;
        choose_layout(est_total, rmax);
        // Layout of a split kernel.  Lanes along the reduce range: the whole block on one output.  Along the outputs:
        // the threads of a row cover 128 contiguous bytes where there are that many outputs.
        auto split_layout = [&](int64_t& l, int64_t& t) {
            l = threads; t = 1;
            if (rc_layout) return;
            const int bytes = reduce_load_bytes(reduces[0]);
            while (t < 128 / bytes && t < total && t < threads) t *= 2;
            l = threads / t;
        };
        if (dyn) { int64_t l, t; split_layout(l, t); lanes = (int)l; touts = (int)t; }

        // Split one long reduction over several blocks?  Where the outputs alone leave SMs idle (fewer than 256 blocks) and a
        // lane makes more than 64 trips: below that the ticket and the second pass over the partials cost what the shorter loop
        // saves.  us split / in one piece: f32 sums of 128 x 128 (64 trips) 3.2 / 2.2, 256 x 256 3.2 / 5.0; over the
        // rows of 1024 x 1024 3.9 / 2.5, 256 x 1024 3.5 / 1.9, 8192 x 8192 (1024 blocks) 52.8 / 47.6, 8192 x 1000 (125 blocks)
        // 10.7 / 14.4, 65536 x 1024 60 / 107.  Each part keeps at least 16 terms a lane (4 wide loads), and the cases of a switch,
        // whose trips are long, are split from there on (a CNN step's weight gradient with 98 trips a lane: the step 76 us split,
        // 87 in one piece).
        // One launch instead of a partials and a finish kernel, whose
        // serial last sum took 2 to 7 us: the loss sum over 8192 x 1000 f16 terms 25 + 6.8 us before.  Over the
        // bound batch, against one block (or one thread) per output: the squared-error sum over 65536 x 1024 f32
        // terms took 167 ms and the column sums of a 65536 x 4096 matrix 3.67 ms; together they are now under
        // 0.4 ms of a 15 ms step (before: 167 ms), and at 256 rows the step went from 740 to 180 us.
        int split = dyn ? -1 : 1;
        if (reduces.size() == 1 && !rsym && !sym_output() && opts.split != 1 && enum_reduce.empty()) {
            if (opts.split > 1) split = opts.split;
            else {
                int64_t lanes_s, touts_s;
                split_layout(lanes_s, touts_s);
                const int64_t nob = (total + touts_s - 1) / touts_s;
                const int64_t s = std::min<int64_t>(rmax / (lanes_s * 16), (148 * 4) / nob);
                const bool long_loop = rmax > (int64_t)lanes * 64 && (total + touts - 1) / touts < 256;
                if (s > 1 && (enum_out.empty() ? long_loop : nob <= 148 * 2)) { split = (int)std::min<int64_t>(s, 1024); lanes = (int)lanes_s; touts = (int)touts_s; }
            }
            if (split > 1 && opts.split > 1) { rc_layout = true; lanes = threads; touts = 1; }
            if (split > 1 && (total + touts - 1) / touts > kMaxTickets) split = 1;
        }
        const int64_t nob = (total + touts - 1) / touts;
        if (dyn && nob > kMaxTickets) return fail("codegen: too many output blocks to split");
        // a switch over output ranges is only safe where the threads that synchronise share the case:
        // no cooperation at all (one lane per output) or one output per block
        if (!enum_out.empty() && !((lanes == 1 && split == 1) || touts == 1)) enum_out.clear();
        split_mode = split != 1;
        split_parts = split;

        reset_emit();
        reduce_combine_mode = "group";
        std::ostringstream k;
        k << reduce_macros(split_mode ? split : 0, nob) << preamble();
        if (split_mode) k << join_preamble();
        std::string name = "reduce_fused";
        k << signature(name, split_mode, threads) << " {\n  enter_();\n";
        k << "  __shared__ float red_smem[" << (rc_layout ? std::max(threads / 32, 1) : threads) << "];\n";
        if (rc_layout) k << "  const int lane = threadIdx.x % LANES, grp = threadIdx.x / LANES;\n";
        else k << "  const int grp = threadIdx.x % TOUTS, lane = threadIdx.x / TOUTS;\n";
        if (split_mode) {
            k << "  __shared__ unsigned split_last;\n";
            k << "  const int ob = blockIdx.x / SPLIT, part = blockIdx.x % SPLIT;\n";
            k << "  long long g = (long long)ob * TOUTS + grp;\n";
        } else k << "  long long g = (long long)blockIdx.x * TOUTS + grp;\n";
        k << "  const bool valid = g < " << total_expr() << ";\n";
        k << "  if (!valid) g = " << total_expr() << " - 1;\n";
        std::string at = "g";                   // place of this thread's output
        if (!enum_reduce.empty() && lanes == 1 && !split_mode && !has_sym) {
            const std::vector<int> order = thread_order(), natural = loop_ranges;
            if (order != natural) {
                loop_ranges = order;
                k << decompose("g");
                loop_ranges = natural;
                at = "";
                int64_t stride = 1;
                for (size_t r = natural.size(); r-- > 0;) { at += (at.empty() ? "r" : " + r") + std::to_string(N(natural[r]).aux) + " * " + std::to_string(stride) + "LL"; stride *= N(natural[r]).arg; }
            }
        }
        if (at == "g") k << decompose("g");
        if (enum_out.empty()) {
            std::string v = val(body, -1);
            if (!err.empty()) return false;
            k << top.code;
            k << "  if (valid && lane == 0) data0[" << at << "] = " << store_value(v, body) << ";\n";
        } else {
            if (!emit_cases(k, "  if (valid && lane == 0) data0[" + at + "] = ")) return false;
        }
        k << "}\n";
        out.klass = split_mode ? KC_REDUCE_SPLIT : KC_REDUCE;
        out.source = k.str();
        out.main.entry = name;
        out.main.block = threads;
        out.main.outputs_per_block = touts;
        out.main.static_outputs = total;
        out.main.sym_trailing = sym_output() ? total : 0;
        out.uses_sym = has_sym;
        if (split_mode) {
            out.split = split;
            out.out_blocks = nob;
            out.part_elems = nob * touts;
            out.split_lanes = lanes;
            if (dyn) { out.sym_terms = 1; for (size_t s2 = 1; s2 < N(reduces[0]).src.size(); s2++) { int rn = N(reduces[0]).src[s2]; if (N(rn).op == OP_RANGE && !N(rn).symbolic()) out.sym_terms *= N(rn).arg; } }
        }
        out.note = std::string("reduce ") + (rc_layout ? "RC" : "OC") + " lanes=" + std::to_string(lanes) + " touts=" + std::to_string(touts);
        if (split_mode) out.note += split > 0 ? " split reduce parts=" + std::to_string(split) : std::string(" split over the bound batch");
        if (!enum_reduce.empty()) out.note += " value-by-value reduce";
        if (!enum_out.empty()) out.note += " switch over " + std::to_string(enum_out.size()) + " output ranges";
        return true;
    }

    // The elementwise kernel `it` as a device function for the contraction kernel's epilogue: eight
    // consecutive outputs of one row at a time, paired f16 arithmetic, the value of parameter
    // `acc_param` at the output position taken from registers instead of memory.  Only kernels the
    // paired-f16 vector path covers qualify; everything else stays a launch of its own.
    bool build_epilogue(int acc_param, int64_t M, int64_t Ncols, EpilogueRendered& out) {
        if (!analyse()) return false;
        if (!reduces.empty() || has_sym) return fail("epilogue: not a static elementwise kernel");
        if (loop_ranges.size() != 2 || N(loop_ranges[0]).arg != M || N(loop_ranges[1]).arg != Ncols) return fail("epilogue: iteration space differs from the contraction's output");
        if (it.bufs[0].dtype != DT_F16 || (int)it.bufs.size() > 8) return fail("epilogue: output is not f16 or too many operands");
        std::vector<int> vloads;
        const int V = pick_vector(vloads);
        if (V != 8 || !h2_eligible(V)) return fail("epilogue: not a paired-f16 vector kernel");
        reset_emit();
        h2 = true;
        const int r0 = loop_ranges[0], r1 = loop_ranges[1];
        bool saw_acc = false;
        cur_top = &prelude;
        int vi = 0;
        std::ostringstream loads;
        for (int i = 0; i < n; i++) {
            if (N(i).op != OP_INDEX || i == dst || !is_live(i)) continue;
            const int p = (int)N(N(i).src[0]).arg;
            if (p != acc_param) continue;
            // must be exactly the contraction's own output position
            Lin f = flat_index(i);
            bool ok0, ok1;
            if (f.c != 0 || f.t.size() != 2 || lin_coef(f, r0, ok0) != Ncols || !ok0 || lin_coef(f, r1, ok1) != 1 || !ok1) return fail("epilogue: the consumer reads the contraction at another position");
            vec_load[i] = "acc";
            saw_acc = true;
        }
        if (!saw_acc) return fail("epilogue: the consumer does not read the contraction");
        for (int i : vloads) {
            if (vec_load.count(i)) continue;
            const int p = (int)N(N(i).src[0]).arg;
            Lin f = flat_index(i);
            // the loads live in a function of their own (epi8_load_), so that the contraction kernel can
            // issue them a chunk ahead of the arithmetic that needs them
            const std::string arr = "v" + std::to_string(vi);
            loads << "  ldv_<__half2, 4>(reinterpret_cast<const __half2*>(data" << p << " + " << render(f, -1) << "), raw[" << vi << "]);\n";
            stmt(-1, "const __half2* " + arr + "_raw = raw[" + std::to_string(vi) + "];");
            vi++;
            vec_load[i] = arr + "_raw";
        }
        cur_top = nullptr;
        vec_range = r1;
        const std::string v = val_h2(body);
        if (!err.empty()) return false;
        std::ostringstream k;
        k << "#define LANES 1\n#define TOUTS 1\n#define RC_LAYOUT 1\n" << preamble();
        std::ostringstream head;
        head << "  const int r" << N(r0).aux << " = row; (void)r" << N(r0).aux << ";\n";
        head << "  const int r" << N(r1).aux << " = col; (void)r" << N(r1).aux << ";\n";
        out.params.clear();
        for (int b = 1; b < (int)it.bufs.size(); b++) {
            if (b == acc_param) continue;
            if (it.bufs[b].dtype != DT_F16) return fail("epilogue: an operand is not f16");
            head << "  const __half* __restrict__ data" << b << " = reinterpret_cast<const __half*>(ep[" << out.params.size() << "]); (void)data" << b << ";\n";
            out.params.push_back(b);
        }
        if (out.params.size() > 6) return fail("epilogue: more than six operands");
        // EPI_NRAW groups of 8 consecutive f16 are loaded per call; raw[k] holds group k as four pairs
        k << "#define EPI_NRAW " << vi << "\n";
        k << "__device__ __forceinline__ void epi8_load_(const int row, const int col, const void* const* ep, __half2 (*raw)[4]) {\n";
        k << head.str() << loads.str() << "}\n";
        k << "__device__ __forceinline__ void epi8_(const int row, const int col, const __half2* __restrict__ acc, __half2* __restrict__ out, const void* const* ep, const __half2 (*raw)[4]) {\n";
        k << head.str();
        k << prelude.code;
        k << "  _Pragma(\"unroll\") for (int u = 0; u < 4; u++) {\n" << top.code << "    out[u] = " << v << ";\n  }\n}\n";
        out.source = k.str();
        out.note = "epilogue of " + std::to_string(out.params.size()) + " operands";
        return true;
    }

    bool opts_untuned() const { return !opts.reduce_lanes && !opts.split; }

    bool run(Rendered& out) {
        if (!analyse()) return false;
        if (it.bufs.empty()) return fail("codegen: kernel has no output buffer");
        if (static_total() >= ((int64_t)1 << 31)) return fail("codegen: more than 2^31 outputs");
        if (opts_untuned()) plan_enumeration();
        bool ok = reduces.empty() ? build_elementwise(out) : build_reduce(out);
        return ok && err.empty();
    }
};

}  // namespace

bool match_contraction(const Item& item, Contraction& c) {
    CodegenOpts o;
    Gen g(item, o);
    if (!g.analyse()) return false;
    if (g.reduces.size() != 1 || g.reduces[0] != g.body) return false;
    const Node& red = g.N(g.body);
    if ((int)red.aux != OP_ADD) return false;
    std::vector<int> rr;
    for (size_t s = 1; s < red.src.size(); s++) if (g.N(red.src[s]).op == OP_RANGE) rr.push_back(red.src[s]);
    if (rr.size() != 1) return false;
    int k = rr[0];
    const Node& mul = g.N(red.src[0]);
    if (mul.op != OP_MUL || mul.src.size() != 2) return false;
    int ia = mul.src[0], ib = mul.src[1];
    if (g.N(ia).op != OP_INDEX || g.N(ib).op != OP_INDEX) return false;
    if (g.loop_ranges.empty() || g.loop_ranges.size() > 3) return false;
    // output = [..m ranges.., n]: n is the innermost loop range read by exactly one operand
    int pa = (int)g.N(g.N(ia).src[0]).arg, pb = (int)g.N(g.N(ib).src[0]).arg;
    if (g.N(g.N(ia).src[0]).op != OP_PARAM || g.N(g.N(ib).src[0]).op != OP_PARAM) return false;
    Lin fa = g.flat_index(ia), fb = g.flat_index(ib);
    if (!g.in_bounds(fa, pa) || !g.in_bounds(fb, pb)) return false;
    auto only_ranges = [&](const Lin& l) { for (auto& t : l.t) if (g.atoms[t.first].kind != Atom::RANGE) return false; return true; };
    if (!only_ranges(fa) || !only_ranges(fb)) return false;
    auto coef = [&](const Lin& l, int r) { bool ok; return g.lin_coef(l, r, ok); };
    // decide which operand carries n (the innermost output range)
    int n_range = g.loop_ranges.back();
    if (coef(fa, n_range) != 0 && coef(fb, n_range) == 0) { std::swap(ia, ib); std::swap(pa, pb); std::swap(fa, fb); }
    if (coef(fa, n_range) != 0 || coef(fb, n_range) == 0) return false;
    // remaining output ranges form M; they must index only A, with nested strides
    // a symbolic extent (the bound batch) may be all of M or all of K; its value arrives at launch
    if (g.N(n_range).symbolic()) return false;
    int64_t M = 1, a_sm = 0;
    c.m_sym = false; c.k_sym = g.N(k).symbolic();
    for (int i = (int)g.loop_ranges.size() - 2; i >= 0; i--) {
        int r = g.loop_ranges[i];
        if (coef(fb, r) != 0) return false;
        int64_t ca = coef(fa, r);
        if (g.N(r).symbolic()) {
            if (g.loop_ranges.size() != 2) return false;
            c.m_sym = true; a_sm = ca; M = 0;
            break;
        }
        if (M == 1) a_sm = ca;
        else if (ca != a_sm * M) return false;
        M *= g.N(r).arg;
    }
    if (g.loop_ranges.size() == 1) { M = 1; a_sm = 0; }
    c.a_param = pa; c.b_param = pb;
    c.M = M; c.N = g.N(n_range).arg; c.K = c.k_sym ? 0 : g.N(k).arg;
    c.a_sm = a_sm; c.a_sk = coef(fa, k); c.a_off = fa.c;
    c.b_sn = coef(fb, n_range); c.b_sk = coef(fb, k); c.b_off = fb.c;
    if (c.a_sk == 0 || c.b_sk == 0 || c.b_sn == 0 || ((M > 1 || c.m_sym) && a_sm == 0)) return false;
    c.in_dtype = item.bufs[pa].dtype;
    if (item.bufs[pb].dtype != c.in_dtype) return false;
    c.out_dtype = item.bufs[0].dtype;
    return true;
}

bool render_gemm_epilogue(const Item& consumer, int acc_param, int64_t M, int64_t N, EpilogueRendered& out, std::string& err) {
    CodegenOpts o;
    Gen g(consumer, o);
    bool ok = g.build_epilogue(acc_param, M, N, out);
    if (!ok) err = g.err.empty() ? "epilogue: rejected" : g.err;
    return ok && g.err.empty();
}

bool match_column_sum(const Item& item, int& src_param, int64_t& rows, int64_t& cols) {
    CodegenOpts o;
    Gen g(item, o);
    if (!g.analyse() || g.has_sym) return false;
    if (g.reduces.size() != 1 || g.reduces[0] != g.body || g.loop_ranges.size() != 1) return false;
    const Node& red = g.N(g.body);
    if ((int)red.aux != OP_ADD || red.dtype != DT_F16 || item.bufs[0].dtype != DT_F16) return false;
    std::vector<int> rr;
    for (size_t s = 1; s < red.src.size(); s++) if (g.N(red.src[s]).op == OP_RANGE) rr.push_back(red.src[s]);
    if (rr.size() != 1) return false;
    const int src = red.src[0];
    if (g.N(src).op != OP_INDEX || g.N(g.N(src).src[0]).op != OP_PARAM) return false;
    const int p = (int)g.N(g.N(src).src[0]).arg;
    if (p < 1 || p >= (int)item.bufs.size() || item.bufs[p].dtype != DT_F16) return false;
    const int64_t n = g.N(g.loop_ranges[0]).arg, m = g.N(rr[0]).arg;
    Lin f = g.flat_index(src);
    bool ok0, ok1;
    if (f.c != 0 || f.t.size() != 2 || g.lin_coef(f, rr[0], ok0) != n || !ok0 || g.lin_coef(f, g.loop_ranges[0], ok1) != 1 || !ok1) return false;
    if (item.bufs[p].elems(0) != m * n) return false;
    src_param = p; rows = m; cols = n;
    return true;
}

bool render_row_chain(const std::vector<const Item*>& items, const std::vector<std::vector<std::pair<int, int>>>& chain_reads,
                      const CodegenOpts& opts, ChainRendered& out, std::string& err) {
    if (items.size() < 2 || chain_reads.size() != items.size()) { err = "chain: needs at least two stages"; return false; }
    // ── can a block hold a whole row in registers?  The row-contiguous operands of all stages, each read from memory
    // once, before the first stage.  Softmax forward + backward over 8192 x 8192 f32 (x and g, 32 registers a thread at
    // 512 threads) went from nine sweeps over L1 and L2 and three exponentials an element to one of each.
    int64_t C = -1;
    std::map<uint32_t, int> row_bufs;                          // buffer id -> dtype, operands held in registers
    std::vector<std::map<int, uint32_t>> row_nodes(items.size());   // stage: INDEX node -> buffer id
    bool held = !opts.debug_bounds;
    int64_t out_bytes = 4;
    for (size_t s = 0; s < items.size() && held; s++) {
        Gen g(*items[s], opts);
        for (auto& pr : chain_reads[s]) g.chain_subst[pr.first] = "x";
        if (!g.analyse() || g.has_sym || g.loop_ranges.empty()) { held = false; break; }
        std::vector<int> loads;
        const int64_t e = g.row_extent(loads);
        if (e == 0 || (e > 0 && C > 0 && e != C)) { held = false; break; }
        if (e > 0) C = e;
        for (int i : loads) {
            const BufDesc& b = items[s]->bufs[(int)g.N(g.N(i).src[0]).arg];
            row_nodes[s][i] = b.id;
            row_bufs[b.id] = b.dtype;
        }
        if (g.loop_ranges.size() == 2) { out_bytes = dt_storage_bytes(items[s]->bufs[0].dtype); if (dtype_cls(items[s]->bufs[0].dtype) != CF32 && dtype_cls(items[s]->bufs[0].dtype) != CF16) held = false; }
    }
    held = held && C > 0 && !row_bufs.empty() && row_bufs.size() <= 3;
    int lanes = 32, vec = 1, chunks = 0, rows_per_block = 1;
    bool shifted = false;
    if (held) {
        bool all16 = true;
        for (auto& b : row_bufs) all16 = all16 && b.second == DT_F16;
        // wide loads from 512 elements on; below that a lane has too few elements for them to matter
        bool all32 = out_bytes == 4;
        for (auto& b : row_bufs) all32 = all32 && b.second == DT_F32;
        if (C >= 512) { if (all16 && out_bytes == 2 && C % 8 == 0) vec = 8; else if (C % 4 == 0 || all32) vec = 4; }
        shifted = C % vec != 0;
        // elements of each operand a lane: 16, or 20 where that halves a block of 256 to 1024 threads (rows of 2049 to 2560,
        // 4097 to 5120 and 8193 to 10240 elements: more blocks an SM, and fewer lanes past the row's end).  us forward + backward, 16 a
        // lane / 20: 8192 x 2052 48.7 / 39.1, 4096 x 9000 109.5 / 94.5, 4096 x 10200 114.7 / 100.5.  Not at 1024 threads,
        // which have 64 registers each.
        const int64_t most = 16;
        auto per_lane = [&](int l) -> int64_t { return l >= 128 && l <= 512 ? 20 : most; };
        // up to 16 elements: one thread a row, which adds them up in the reference's order, like the separate kernels do
        if (C <= most) lanes = 1;
        const int64_t span = C + (shifted ? vec - 1 : 0);
        while (lanes < 1024 && lanes * per_lane(lanes) < span) lanes *= 2;
        if (lanes * per_lane(lanes) < span) held = false;
        chunks = (int)((span + (int64_t)lanes * vec - 1) / ((int64_t)lanes * vec));
        if (lanes <= 32) rows_per_block = 128 / lanes;        // a warp a row needs no barrier, so rows share a block
    }
    // Long rows, many of them: the blocks stay and walk the rows, and while one row is worked on, each thread already
    // copies its own elements of the next into its own place in shared memory (cp.async, no barrier).  A block that
    // only loads between rows leaves memory idle during its five reductions: softmax forward + backward took 151 us for
    // 8192 x 8192 and 47 for 3001 x 4999 with the rows in registers alone, 137 and 38 this way.
    int64_t row_bytes = 0;
    if (held) for (auto& b : row_bufs) row_bytes += (int64_t)chunks * vec * lanes * dt_storage_bytes(b.second);
    bool piped = held && lanes >= 128 && row_bytes <= 200 * 1024;
    for (auto& b : row_bufs) if (vec * dt_storage_bytes(b.second) < 4) piped = false;
    auto shift_decl = [&](const char* r) { return shifted ? "  const int shift = (int)(((long long)" + std::string(r) + " * " + std::to_string(C) + "LL) & " + std::to_string(vec - 1) + ");\n" : std::string(); };
    const int threads = held ? lanes * rows_per_block : opts.block_threads > 0 ? opts.block_threads : 512;
    std::ostringstream k, sig, body, aligned, loads, fetch, take;      // of the rows: plain loads, or fetch to shared memory and take from there
    int64_t smem_at = 0;
    std::vector<std::string> result(items.size());
    std::vector<bool> inner(items.size(), false);
    int64_t rows = -1;
    int segments = 0;
    // Ask for as many blocks an SM as the registers allow: 16 and half as many again as the row's elements for the
    // values that sweeps share.  Where the row stays in memory, full occupancy (2048 threads per SM): without that bound
    // the run-time compiler took 36 registers for an 8192-wide softmax chain and one of four resident blocks was lost.
    int blocks = threads <= 1024 && 2048 % threads == 0 ? 2048 / threads : 0;
    if (held) {
        int regs = 0;
        for (auto& b : row_bufs) regs += chunks * vec * dt_storage_bytes(b.second) / 4;
        blocks = std::max(1, std::min({65536 / (threads * (24 + regs + regs / 4)), 2048 / threads, 16}));
        if (piped) blocks = (int)std::max<int64_t>(1, std::min<int64_t>(blocks, 227 * 1024 / (row_bytes + 6 * 1024)));
        const int64_t rows0 = items[0]->bufs[0].shape.empty() ? 1 : items[0]->bufs[0].shape[0];
        if (rows0 < 2 * 148 * blocks) piped = false;
    }
    sig << "extern \"C\" __global__ void __launch_bounds__(" << threads;
    if (blocks > 0) sig << ", " << blocks;
    sig << ") row_chain(";
    bool first_arg = true, sweeps = false;
    std::string decls;
    std::map<uint32_t, std::string> reg_name;
    for (size_t s = 0; s < items.size(); s++) {
        Gen g(*items[s], opts);
        for (auto& pr : chain_reads[s]) {
            if (pr.second < 0 || pr.second >= (int)s || inner[pr.second]) { err = "chain: stage input is not a per-row result of an earlier stage"; return false; }
            g.chain_subst[pr.first] = result[pr.second];
        }
        if (held) {
            g.row_len = C; g.row_shifted = shifted; g.row_vec = vec; g.row_chunks = chunks; g.row_slot = &segments;
            for (auto& nb : row_nodes[s]) {
                const int p = (int)g.N(g.N(nb.first).src[0]).arg;
                auto f = reg_name.find(nb.second);
                if (f == reg_name.end()) {
                    // loaded before the first stage, through this stage's pointer
                    const std::string nm = "row" + std::to_string(reg_name.size()), bt = buf_ctype(items[s]->bufs[p].dtype), V = std::to_string(vec);
                    f = reg_name.insert({nb.second, nm}).first;
                    const int esz = dt_storage_bytes(items[s]->bufs[p].dtype), bytes = vec * esz;
                    const std::string src = "s" + std::to_string(s) + "_data" + std::to_string(p);
                    loads << "  " << bt << " " << nm << "[" << chunks * vec << "];\n";
                    for (int c = 0; c < chunks; c++) {
                        const std::string cb = "((" + std::to_string(c * lanes) + " + lane)" + (vec > 1 ? " * " + V : std::string()) + (shifted ? " - shift)" : ")");
                        // a shifted chunk may start up to 3 elements before the row and end as far behind it: inside the
                        // 16-byte group either way, and blocks of device memory are whole 256-byte units
                        const bool all = (int64_t)(c + 1) * lanes * vec <= C;
                        const std::string at = nm + " + " + std::to_string(c * vec), live = all ? std::string() : "if (" + cb + " < " + std::to_string(C) + ") ";
                        std::string zero;
                        for (int u = 0; u < vec; u++) zero += nm + "[" + std::to_string(c * vec + u) + "] = " + (bt == "float" ? "0.0f" : "__float2half_rn(0.0f)") + "; ";
                        if (piped) {
                            const std::string place = "staged + " + std::to_string(smem_at + (int64_t)c * lanes * bytes) + " + lane * " + std::to_string(bytes);
                            fetch << "    " << live << "fetch_<" << bytes << ">(" << place << ", " << src << " + (long long)next * " << C << "LL + " << cb << ");\n";
                            take << "  " << live << "take_<" << bt << ", " << V << ">(" << place << ", " << at << ");" << (all ? std::string() : " else { " + zero + "}") << "\n";
                        } else {
                            loads << "  " << live;
                            if (vec > 1) loads << "ldv_<" << bt << ", " << V << ">(" << src << " + (long long)row * " << C << "LL + " << cb << ", " << at << ");";
                            else loads << nm << "[" << c << "] = __ldg(" << src << " + (long long)row * " << C << "LL + " << cb << ");";
                            loads << (all ? std::string() : " else { " + zero + "}") << "\n";
                        }
                    }
                    smem_at += (int64_t)chunks * lanes * bytes;
                }
                g.row_reg[nb.first] = f->second;
            }
        }
        std::string decl, code; int64_t r = 0; bool has_inner = false;
        if (!g.build_chain_stage((int)s, held ? lanes : threads, decl, code, result[s], r, has_inner)) { err = g.err.empty() ? "chain: stage rejected" : g.err; return false; }
        if (rows >= 0 && r != rows) { err = "chain: stages iterate different row counts"; return false; }
        rows = r;
        inner[s] = has_inner;
        sweeps = sweeps || has_inner || !g.reduces.empty();
        if (has_inner && s + 1 != items.size()) { err = "chain: only the last stage may produce a full row"; return false; }
        decls += decl;
        body << code;
        if (piped && s == 0) body << "  @NEXT@\n";
        for (size_t b = 0; b < items[s]->bufs.size(); b++) {
            // written by this kernel: never const, and not restrict either, as two stages' results may share memory
            std::string ty = b == 0 ? std::string(buf_ctype(items[s]->bufs[b].dtype)) + "*" : "const " + std::string(buf_ctype(items[s]->bufs[b].dtype)) + "* __restrict__";
            sig << (first_arg ? "" : ", ") << ty << " s" << s << "_data" << b << "_";
            // device blocks are 256-byte aligned (pool granularity, 128-element view offsets)
            const std::string local = "s" + std::to_string(s) + "_data" + std::to_string(b);
            aligned << "  " << ty << " " << local << " = (" << ty << ")__builtin_assume_aligned(" << local << "_, 16); (void)" << local << ";\n";
            first_arg = false;
        }
    }
    // one value a row each and nothing to run along the row: plain elementwise kernels, a thread a value, not a block
    // (eight independent products of 100000 values: 8.2 us each in one chain, 1.9 as kernels of their own)
    if (!sweeps) { err = "chain: no stage runs along the row"; return false; }
    sig << ")";
    k << "#define LANES " << (held ? lanes : threads) << "\n#define TOUTS 1\n#define RC_LAYOUT 1\n";
    k << "#define RED_BEGIN(n) lane\n#define RED_END(n) (n)\n#define RED_STEP LANES\n";
    k << Gen::preamble();
    if (held) k << Gen::row_preamble();
    k << sig.str() << " {\n  enter_();\n";
    k << "  __shared__ float red_smem[" << (held ? 32 * std::max(segments, 1) : std::max(threads / 32, 1)) << "];\n";
    if (rows_per_block > 1) {
        k << "  const int lane = threadIdx.x % LANES, row = blockIdx.x * " << rows_per_block << " + threadIdx.x / LANES;\n";
        k << "  if (row >= " << rows << ") return;\n";
    } else if (piped) {
        k << "  extern __shared__ __align__(16) unsigned char staged[];\n  const int lane = threadIdx.x;\n";
    } else {
        k << "  const int lane = threadIdx.x, grp = 0;\n  (void)grp;\n";
        k << "  const int row = blockIdx.x;\n";
    }
    k << "  (void)red_smem;\n" << aligned.str();
    std::string stages = decls + body.str();
    if (piped) {
        // The next row is asked for after the first stage.  A thread copies into the place that it alone has read, and its
        // reads come first in program order: those of operands that the first stage uses have arrived by then, the others
        // rest on that order.
        k << "  { const int next = blockIdx.x;\n" << shift_decl("next") << fetch.str() << "  }\n";
        const size_t at = stages.find("@NEXT@");
        stages = stages.substr(0, at) + "if (row + (int)gridDim.x < " + std::to_string(rows) + ") { const int next = row + (int)gridDim.x;\n" + shift_decl("next") + fetch.str() + "  }\n" + stages.substr(at + 6);
        k << "  for (int row = blockIdx.x; row < " << rows << "; row += gridDim.x) {\n  fetched_();\n" << shift_decl("row") << loads.str() << take.str() << stages;
        if (segments < 2) k << "  __syncthreads();\n";            // with two reductions, either's barrier keeps the other's segment
        k << "  }\n}\n";
    } else k << shift_decl("row") << loads.str() << stages << "}\n";
    out.full_row = inner.back();
    out.own_row.assign(items.size(), {});
    for (size_t s = 0; s < items.size(); s++) {
        Gen g(*items[s], opts);
        if (!g.analyse()) { err = g.err; return false; }
        for (size_t b = 0; b < items[s]->bufs.size(); b++)
            out.own_row[s].push_back(out.full_row && b > 0 && rows > 0 && g.reads_own_row((int)b, items.back()->bufs[0].elems(0) / rows));
    }
    out.blocks_per_sm = piped ? blocks : 0;
    out.smem_bytes = piped ? (unsigned)smem_at : 0u;
    out.source = k.str();
    out.block = (unsigned)threads;
    out.rows = rows;
    out.rows_per_block = rows_per_block;
    out.held = held;
    out.note = "row chain of " + std::to_string(items.size()) + " stages, " + std::to_string(rows) + " rows";
    if (held) out.note += ", " + std::to_string(row_bufs.size()) + " operands in registers, " + std::to_string(lanes) + " lanes a row";
    return true;
}

bool chain_overwrites(const std::vector<const Item*>& items, const std::vector<std::vector<std::pair<int, int>>>& chain_reads,
                      const ChainRendered& r, const std::function<int(const BufDesc&, const BufDesc&)>& place) {
    auto alike = [](const BufDesc& a, const BufDesc& b) { return a.dtype == b.dtype && a.elems(0) == b.elems(0); };
    for (size_t w = 0; w < items.size(); w++) {
        const BufDesc& o = items[w]->bufs[0];
        const bool full = r.full_row && w + 1 == items.size();
        // two results: a value a row each, one over the other, is written by the same thread in order
        for (size_t v = 0; v < w; v++) {
            const int at = place(o, items[v]->bufs[0]);
            if (at && (at != 1 || full || !alike(o, items[v]->bufs[0]))) return true;
        }
        // A result over an operand: only a whole row over the very elements that the same row has been read from.  A value
        // a row would need the operand read at the row's index, and by all threads before the first of them stores.
        for (size_t m = 0; m < items.size(); m++)
            for (size_t b = 1; b < items[m]->bufs.size(); b++) {
                const BufDesc& in = items[m]->bufs[b];
                bool from_register = false;
                for (auto& pr : chain_reads[m]) from_register = from_register || pr.first == (int)b;
                if (from_register || o.id == in.id) continue;
                const int at = place(o, in);
                if (at && !(at == 1 && full && alike(o, in) && r.own_row[m][b])) return true;
            }
    }
    return false;
}

bool render_cuda(const Item& item, const CodegenOpts& opts, Rendered& out, std::string& err) {
    Gen g(item, opts);
    bool ok = g.run(out);
    if (!ok) err = g.err.empty() ? "codegen: failed" : g.err;
    return ok;
}

}  // namespace anl
