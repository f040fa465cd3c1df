// llg_blockplan.cpp -- plans a gate list as dense 5-qubit blocks (llg_gateblock.cu) for 16-byte
// states of 6 and more qubits.
//
// A block costs the same whatever it holds, so the plan wants few of them.  Runs of one-qubit gates
// are multiplied first (g2 @ g1).  Order is kept per qubit, up to commutation in the Z basis: a
// qubit's gates form segments, each a maximal run of gates that are diagonal on it (RZ, CZ / MCZ, a
// CNOT's control), in any order, or one gate that is not.  A gate is ready when it is in the current
// segment of each of its qubits.
//
// Greedy: for a few of the earliest ready gates as seeds, the qubit set starts with the seed's
// qubits and grows to five, each time by the qubit that lets the block absorb most (every ready gate
// inside the set, repeatedly); the best seed's block is emitted.  On the layered-rotation circuit
// this packs a layer of 30 qubits into 2.9 blocks (an exhaustive choice among all seeds: the same).
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <string>
#include <vector>

#include "llg_internal.h"

namespace llg {

namespace {

struct Node {
    uint64_t mask = 0;  // its qubits
    int kind = 0;       // BlockGate kinds
    int mat = -1;       // kind 0: its 2x2 matrix; kind 1: the target; kind 3: its occurrence; kind 4: its index
    int axis = 0;       // kind 3
    int seg_begin = 0;  // its qubits in increasing order: segments seg_of_[seg_begin ..]
    float weight = 0.f;
};

void matmul(const double* a, const double* b, double* out) {
    using cd = std::complex<double>;
    const cd a0(a[0], a[1]), a1(a[2], a[3]), a2(a[4], a[5]), a3(a[6], a[7]);
    const cd b0(b[0], b[1]), b1(b[2], b[3]), b2(b[4], b[5]), b3(b[6], b[7]);
    const cd r[4] = {a0 * b0 + a1 * b2, a0 * b1 + a1 * b3, a2 * b0 + a3 * b2, a2 * b1 + a3 * b3};
    for (int k = 0; k < 4; ++k) {
        out[2 * k] = r[k].real();
        out[2 * k + 1] = r[k].imag();
    }
}

// what a 2x2 costs in tile passes; a run of them by the classes alone
enum Class2x2 : uint8_t { kNone, kDiag, kMove, kH, kRealX, kRealY, kGeneral, kClasses };
constexpr Class2x2 kMerge[kClasses][kClasses] = {
    {kNone, kDiag, kMove, kH, kRealX, kRealY, kGeneral},
    {kDiag, kDiag, kMove, kGeneral, kGeneral, kGeneral, kGeneral},
    {kMove, kMove, kDiag, kGeneral, kGeneral, kGeneral, kGeneral},
    {kH, kGeneral, kGeneral, kNone, kGeneral, kGeneral, kGeneral},
    {kRealX, kGeneral, kGeneral, kGeneral, kRealX, kGeneral, kGeneral},
    {kRealY, kGeneral, kGeneral, kGeneral, kGeneral, kRealY, kGeneral},
    {kGeneral, kGeneral, kGeneral, kGeneral, kGeneral, kGeneral, kGeneral},
};
Class2x2 class_2x2(const double* m) {
    auto zero = [&](int k) { return m[2 * k] == 0.0 && m[2 * k + 1] == 0.0; };
    if (zero(1) && zero(2)) return kDiag;
    if (zero(0) && zero(3)) return kMove;
    if (m[1] != 0.0 || m[7] != 0.0) return kGeneral;
    if (m[3] == 0.0 && m[5] == 0.0) return m[0] == m[2] && m[0] == m[4] && m[0] == -m[6] ? kH : kRealY;
    return m[2] == 0.0 && m[4] == 0.0 ? kRealX : kGeneral;
}
// of the named one-qubit gates, by kind
constexpr Class2x2 kNamed[] = {kH, kMove, kRealX, kRealY, kDiag};
static_assert(LLG_OP_H == 0 && LLG_OP_X == 1 && LLG_OP_RX == 2 && LLG_OP_RY == 3 && LLG_OP_RZ == 4, "kNamed's order");
// log2 of the smallest entry of a 2x2 that mixes where that is below 2^-7, else 0 (entries below 2^-50 are roundings of 0)
float small_entry(const double* m) {
    double least = 1.0;
    for (int k = 0; k < 4; ++k) {
        const double n2 = m[2 * k] * m[2 * k] + m[2 * k + 1] * m[2 * k + 1];
        if (n2 > 0x1p-100) least = std::min(least, n2);
    }
    return least < 0x1p-14 ? 0.5f * (float)std::log2(least) : 0.0f;
}
void add_classes(const int* count, GateCounts& c) {
    c.diag += count[kDiag];
    c.moves += count[kMove];
    c.h += count[kH];
    c.real += count[kRealX] + count[kRealY];
    c.general += count[kGeneral];
}

}  // namespace

GateCounts count_gates(int n, const llg_op* ops, int nops, const std::vector<MatrixOp>& matrices, int* two, double* partners) {
    GateCounts c;
    Class2x2 open[64];
    uint64_t met[64];
    int count[kClasses] = {};
    for (int q = 0; q < n; ++q) {
        open[q] = kNone;
        met[q] = 0;
    }
    auto close = [&](int q, uint64_t mask) {
        ++count[open[q]];
        open[q] = kNone;
        met[q] |= mask;
    };
    *two = 0;
    for (int i = 0; i < nops; ++i) {
        const llg_op& o = ops[i];
        if (o.kind <= LLG_OP_RZ) {
            open[o.q0] = kMerge[open[o.q0]][kNamed[o.kind]];
        } else if (o.kind == LLG_OP_CNOT || o.kind == LLG_OP_CZ) {
            const uint64_t mask = 1ULL << o.q0 | 1ULL << o.q1;
            close(o.q0, mask);
            close(o.q1, mask);
            ++*(o.kind == LLG_OP_CNOT ? &c.moves : &c.flips);
            ++*two;
        } else if (o.kind == LLG_OP_MCZ) {
            for (uint64_t s = o.mask; s; s &= s - 1) close(__builtin_ctzll(s), o.mask);
            ++c.flips;
            ++*two;
        } else if (o.kind == kOpMatrix) {
            const MatrixOp& m = matrices[o.q0];
            uint64_t mask = 0;
            for (int j = 0; j < m.k; ++j) mask |= 1ULL << m.q[j];
            for (int j = 0; j < m.k; ++j) close(m.q[j], mask);
            ++(m.k <= 2 ? c.small : c.large);
        } else {
            open[o.q0] = kMerge[open[o.q0]][class_2x2(o.m)];
        }
    }
    int pairs = 0;
    for (int q = 0; q < n; ++q) {
        close(q, 0);
        pairs += met[q] ? __builtin_popcountll(met[q]) - 1 : 0;
    }
    add_classes(count, c);
    *partners = (double)pairs / n;
    return c;
}

class BlockPlanner::Impl {
public:
    Impl(int n, const llg_op* ops, int nops, bool params, const std::vector<MatrixOp>* matrices, BlockPlan& out)
        : n_(n), params_(params), mops_(matrices), out_(out) {
        build(ops, nops);
    }

    bool advance(int blocks) {
        const int goal = out_.blocks + blocks;
        while (remaining_ > 0 && out_.blocks < goal) {
            if (wide_ > 0 && emit_wide()) continue;
            emit(choose());
        }
        return remaining_ > 0;
    }

    void mark() { marked_ = done_; }

    std::vector<llg_op> rest(const llg_op* ops, int nops) const {
        std::vector<llg_op> r;
        for (int i = 0; i < nops; ++i) {
            const int id = op_node_[i] < 0 ? node_of_mat_[-1 - op_node_[i]] : op_node_[i];
            if (!marked_[id]) r.push_back(ops[i]);
        }
        return r;
    }

private:
    struct M8 {
        double m[8];
    };
    static bool wide(const Node& v) { return __builtin_popcountll(v.mask) > 5; }

    // appends a gate; zmask: the qubits it is diagonal on
    void add_node(Node v, uint64_t zmask) {
        const int id = (int)nodes_.size();
        v.seg_begin = (int)seg_of_.size();
        for (uint64_t s = v.mask; s; s &= s - 1) {
            const int q = __builtin_ctzll(s);
            const bool z = zmask >> q & 1;
            std::vector<int>& b = seg_start_[q];
            if (b.empty() || !z || !last_z_[q]) b.push_back((int)ids_[q].size());
            last_z_[q] = z;
            ids_[q].push_back(id);
            seg_of_.push_back((int)b.size() - 1);
        }
        if (wide(v)) ++wide_;
        nodes_.push_back(v);
    }

    void build(const llg_op* ops, int nops) {
        std::vector<int> pend(n_, -1);  // index into mats_ of the open run of one-qubit gates
        std::vector<char> pdiag(n_, 0);
        nodes_.reserve(nops);
        mats_.reserve(nops);
        node_of_mat_.reserve(nops);
        seg_of_.reserve(2 * nops);
        op_node_.resize(nops);
        for (int q = 0; q < n_; ++q) {
            ids_[q].reserve((size_t)nops / n_ + 8);
            seg_start_[q].reserve((size_t)nops / n_ + 8);
        }
        auto flush = [&](int q) {
            if (pend[q] < 0) return;
            node_of_mat_[pend[q]] = (int)nodes_.size();
            Node v;
            v.mask = 1ULL << q;
            v.mat = pend[q];
            v.weight = pdiag[q] ? 0.5f : 1.0f;
            add_node(v, pdiag[q] ? v.mask : 0);
            pend[q] = -1;
        };
        int occ = 0;
        for (int i = 0; i < nops; ++i) {
            const llg_op& op = ops[i];
            if (params_ && op.param >= 0) {
                flush(op.q0);
                Node v;
                v.kind = 3;
                v.mask = 1ULL << op.q0;
                v.mat = occ++;
                v.axis = op.kind == LLG_OP_RX ? 0 : (op.kind == LLG_OP_RY ? 1 : 2);
                v.weight = v.axis == 2 ? 0.5f : 1.0f;
                op_node_[i] = (int)nodes_.size();
                add_node(v, v.axis == 2 ? v.mask : 0);
                continue;
            }
            if (is_single_qubit(op.kind)) {
                M8 g;
                op_matrix(op, g.m);
                const bool d = g.m[2] == 0.0 && g.m[3] == 0.0 && g.m[4] == 0.0 && g.m[5] == 0.0;
                if (pend[op.q0] < 0) {
                    pend[op.q0] = (int)mats_.size();
                    mats_.push_back(g);
                    node_of_mat_.push_back(-1);
                    pdiag[op.q0] = d;
                } else {
                    M8& p = mats_[pend[op.q0]];
                    matmul(g.m, p.m, p.m);
                    pdiag[op.q0] = pdiag[op.q0] && d;
                }
                op_node_[i] = -1 - pend[op.q0];
                continue;
            }
            if (op.kind == kOpMatrix) {
                const MatrixOp& mo = (*mops_)[op.q0];
                Node v;
                v.kind = 4;
                v.mat = op.q0;
                for (int j = 0; j < mo.k; ++j) v.mask |= 1ULL << mo.q[j];
                for (uint64_t s = v.mask; s; s &= s - 1) flush(__builtin_ctzll(s));
                bool diag = true;
                const int d = 1 << mo.k;
                for (int e = 0; e < d * d; ++e)
                    if (e / d != e % d) diag = diag && mo.m[2 * e] == 0.0 && mo.m[2 * e + 1] == 0.0;
                v.weight = mo.k <= 2 ? 2.0f : 5.0f;
                op_node_[i] = (int)nodes_.size();
                add_node(v, diag ? v.mask : 0);
                continue;
            }
            Node v;
            v.weight = 0.6f;
            v.kind = op.kind == LLG_OP_CNOT ? 1 : 2;
            v.mask = op.kind == LLG_OP_MCZ ? op.mask : (1ULL << op.q0 | 1ULL << op.q1);
            for (uint64_t s = v.mask; s; s &= s - 1) flush(__builtin_ctzll(s));
            uint64_t z = v.mask;
            if (v.kind == 1) {
                v.mat = op.q1;
                z = 1ULL << op.q0;
            }
            op_node_[i] = (int)nodes_.size();
            add_node(v, z);
        }
        for (int q = 0; q < n_; ++q) {
            flush(q);
            seg_start_[q].push_back((int)ids_[q].size());  // end of the last segment
        }
        remaining_ = (int)nodes_.size();
        stamp_.assign(nodes_.size(), 0);
        done_.assign(nodes_.size(), 0);
        for (int q = 0; q < n_; ++q) {
            cur_[q] = 0;
            left_[q] = segs(q) > 0 ? seg_size(q, 0) : 0;
        }
    }

    int segs(int q) const { return (int)seg_start_[q].size() - 1; }
    int seg_size(int q, int s) const { return seg_start_[q][s + 1] - seg_start_[q][s]; }

    bool ready(const Node& v, const int* cur) const {
        int k = v.seg_begin;
        for (uint64_t s = v.mask; s; s &= s - 1, ++k)
            if (cur[__builtin_ctzll(s)] != seg_of_[k]) return false;
        return true;
    }

    // What a block has taken so far: the current segment of each of its qubits and the gates (marked
    // with `stamp`).  Growing the set only adds gates, so a larger set starts from the smaller one's.
    struct Taken {
        uint64_t set = 0;
        double weight = 0.0;
        int cur[64], left[64];
    };

    // adds qubit(s) `add` to the block and takes every gate that becomes possible; gates are marked
    // with `stamp` (those of the smaller set carry `base`)
    void extend(Taken& t, uint64_t add, int base, int stamp, std::vector<int>* got) {
        uint64_t work = add;  // qubits whose current segment is new
        for (uint64_t s = add; s; s &= s - 1) {
            const int q = __builtin_ctzll(s);
            t.cur[q] = cur_[q];
            t.left[q] = left_[q];
        }
        t.set |= add;
        while (work) {
            const int q = __builtin_ctzll(work);
            work &= work - 1;
            const int seg = t.cur[q];
            if (seg >= segs(q)) continue;
            for (int i = seg_start_[q][seg]; i < seg_start_[q][seg + 1]; ++i) {
                const int id = ids_[q][i];
                if (done_[id] || stamp_[id] == stamp || stamp_[id] == base) continue;
                const Node& v = nodes_[id];
                if ((v.mask & ~t.set) || !ready(v, t.cur)) continue;
                stamp_[id] = stamp;
                if (got) got->push_back(id);
                t.weight += v.weight;
                for (uint64_t s = v.mask; s; s &= s - 1) {
                    const int p = __builtin_ctzll(s);
                    if (--t.left[p] == 0) {
                        const int ns = ++t.cur[p];
                        t.left[p] = ns < segs(p) ? seg_size(p, ns) : 0;
                        work |= 1ULL << p;
                    }
                }
                if (t.cur[q] != seg) break;
            }
        }
    }

    // qubits of gates that touch the block and would be next
    uint64_t partners(const Taken& t, int stamp) const {
        uint64_t p = 0;
        for (uint64_t s = t.set; s; s &= s - 1) {
            const int q = __builtin_ctzll(s), seg = t.cur[q];
            if (seg >= segs(q)) continue;
            for (int i = seg_start_[q][seg]; i < seg_start_[q][seg + 1]; ++i) {
                const int id = ids_[q][i];
                if (!done_[id] && stamp_[id] != stamp && !wide(nodes_[id])) p |= nodes_[id].mask & ~t.set;
            }
        }
        return p;
    }

    // an MCZ on more than five qubits that is ready runs on its own
    bool emit_wide() {
        bool any = false;
        for (size_t id = first_; id < nodes_.size(); ++id) {
            const Node& v = nodes_[id];
            if (done_[id] || !wide(v) || !ready(v, cur_)) continue;
            finish((int)id);
            single(v);
            --wide_;
            any = true;
        }
        return any;
    }

    void finish(int id) {
        done_[id] = 1;
        --remaining_;
        for (uint64_t s = nodes_[id].mask; s; s &= s - 1) {
            const int q = __builtin_ctzll(s);
            if (--left_[q] == 0) {
                const int ns = ++cur_[q];
                left_[q] = ns < segs(q) ? seg_size(q, ns) : 0;
            }
        }
        while (first_ < nodes_.size() && done_[first_]) ++first_;
    }

    // grows a set of at most five qubits around `seed`
    void grow(uint64_t seed, Taken& t) {
        t.set = 0;
        t.weight = 0.0;
        const int base = ++stamp_id_;
        extend(t, seed, base, base, nullptr);
        while (__builtin_popcountll(t.set) < std::min(5, n_)) {
            uint64_t cand = partners(t, base);
            if (!cand) {  // nothing connected is next: a few of the qubits that still have gates
                int c = 0;
                for (int q = 0; q < n_ && c < 6; ++q)
                    if (!(t.set >> q & 1) && cur_[q] < segs(q)) {
                        cand |= 1ULL << q;
                        ++c;
                    }
            }
            if (!cand) break;
            double bw = -1.0;
            uint64_t bq = 0;
            for (uint64_t s = cand; s; s &= s - 1) {
                const uint64_t bit = s & -s;
                try_.weight = t.weight;
                try_.set = t.set;
                for (uint64_t r = t.set; r; r &= r - 1) {
                    const int q = __builtin_ctzll(r);
                    try_.cur[q] = t.cur[q];
                    try_.left[q] = t.left[q];
                }
                extend(try_, bit, base, ++stamp_id_, nullptr);
                if (try_.weight > bw) {
                    bw = try_.weight;
                    bq = bit;
                }
            }
            extend(t, bq, base, base, nullptr);
        }
    }

    uint64_t choose() {
        uint64_t seen[kSeeds], best = 0;
        int ns = 0;
        double bw = -1.0;
        for (size_t id = first_; id < nodes_.size() && ns < kSeeds; ++id) {
            const Node& v = nodes_[id];
            if (done_[id] || wide(v) || !ready(v, cur_)) continue;
            bool dup = false;
            for (int k = 0; k < ns; ++k) dup |= (v.mask & ~seen[k]) == 0;  // inside a tried block
            if (dup) continue;
            grow(v.mask, tried_);
            seen[ns++] = tried_.set;
            if (tried_.weight > bw) {
                bw = tried_.weight;
                best = tried_.set;
            }
        }
        return best;
    }

    void gate(const Node& v, const int* to_local) {
        out_.gates.emplace_back();
        BlockGate& g = out_.gates.back();
        std::memset(&g, 0, sizeof(g));
        g.kind = v.kind;
        auto local = [&](int q) { return to_local ? to_local[q] : q; };
        if (v.kind == 4) {
            const MatrixOp& mo = (*mops_)[v.mat];
            for (int j = 0; j < mo.k; ++j) g.q0 |= local(mo.q[j]) << (4 * j);
            g.q1 = mo.k;
            g.pad = (int)(out_.matrices.size() / 2);
            out_.matrices.insert(out_.matrices.end(), mo.m.begin(), mo.m.end());
            ++(mo.k <= 2 ? out_.counts.small : out_.counts.large);
        } else if (v.kind == 3) {
            g.q0 = local(__builtin_ctzll(v.mask));
            g.q1 = v.mat;
            g.pad = v.axis;
        } else if (v.kind == 0) {
            const Class2x2 cls = class_2x2(mats_[v.mat].m);
            int count[kClasses] = {};
            count[cls] = 1;
            add_classes(count, out_.counts);
            if (cls != kDiag && cls != kMove) {
                float& most = small_[local(__builtin_ctzll(v.mask))];
                most = std::max(most, small_entry(mats_[v.mat].m));
            }
            g.q0 = local(__builtin_ctzll(v.mask));
            std::memcpy(g.m, mats_[v.mat].m, sizeof(g.m));
        } else if (v.kind == 1) {
            ++out_.counts.moves;
            g.q0 = local(__builtin_ctzll(v.mask & ~(1ULL << v.mat)));
            g.q1 = local(v.mat);
        } else {
            ++out_.counts.flips;
            for (uint64_t s = v.mask; s; s &= s - 1) g.mask |= 1ULL << local(__builtin_ctzll(s));
        }
    }

    void single(const Node& v) {
        BlockStep st;
        std::memset(&st, 0, sizeof(st));
        st.gate_begin = (int)out_.gates.size();
        st.ngates = 1;
        gate(v, nullptr);
        out_.steps.push_back(st);
    }

    void emit(uint64_t set) {
        got_.clear();
        Taken& t = tried_;
        t.set = 0;
        t.weight = 0.0;
        const int id0 = ++stamp_id_;
        extend(t, set, id0, id0, &got_);
        for (int id : got_) finish(id);
        // up to three gates that only move amplitudes or signs run on their own: a CNOT or CZ pass
        // takes 2.6 ms at 30 qubits, a block 8.8
        bool moves = !params_ && got_.size() <= 3;
        for (int id : got_) moves = moves && (nodes_[id].kind == 1 || nodes_[id].kind == 2);
        if (moves) {
            for (int id : got_) single(nodes_[id]);
            return;
        }
        for (int q = n_ - 1; q >= 0 && __builtin_popcountll(set) < 5; --q) set |= 1ULL << q;
        BlockStep st;
        std::memset(&st, 0, sizeof(st));
        st.is_block = 1;
        int to_local[64];
        int k = 0;
        for (uint64_t s = set; s; s &= s - 1) {
            const int q = __builtin_ctzll(s);
            st.q[k] = q;
            to_local[q] = k++;
        }
        st.gate_begin = (int)out_.gates.size();
        st.ngates = (int)got_.size();
        constexpr float kUnset = -1e9f;  // no gate that mixes
        for (int b = 0; b < 5; ++b) small_[b] = kUnset;
        for (int id : got_) gate(nodes_[id], to_local);
        out_.steps.push_back(st);
        ++out_.blocks;
        float bits = 0.0f;
        for (int b = 0; b < 5; ++b) bits += small_[b] > kUnset ? small_[b] : 0.0f;
        out_.fades = out_.fades || bits < -44.0f;
    }

    static constexpr int kSeeds = 4;
    int n_;
    bool params_;
    const std::vector<MatrixOp>* mops_;
    BlockPlan& out_;
    std::vector<M8> mats_;
    std::vector<Node> nodes_;
    std::vector<int> seg_of_;
    std::vector<int> op_node_, node_of_mat_;  // per op: its node, or -1 less the index of its run's matrix
    std::vector<int> ids_[64], seg_start_[64];  // per qubit: its gates in order, where each segment starts
    bool last_z_[64] = {};
    int cur_[64], left_[64];  // per qubit: the current segment, its gates not done yet
    std::vector<int> stamp_, got_;
    std::vector<char> done_, marked_;
    Taken tried_, try_;
    float small_[64] = {};  // per qubit of the block: small_entry of the gate that mixes most
    int stamp_id_ = 0, remaining_ = 0, wide_ = 0;
    size_t first_ = 0;
};

BlockPlanner::BlockPlanner(int n, const llg_op* ops, int nops, bool params, const std::vector<MatrixOp>* matrices)
    : impl_(new Impl(n, ops, nops, params, matrices, plan)) {}
BlockPlanner::~BlockPlanner() = default;
bool BlockPlanner::advance(int blocks) { return impl_->advance(blocks); }
void BlockPlanner::mark() { impl_->mark(); }
std::vector<llg_op> BlockPlanner::rest(const llg_op* ops, int nops) const { return impl_->rest(ops, nops); }

double spectral_norm_2x2(const double* m) {
    double f2 = 0.0;
    for (int k = 0; k < 8; ++k) f2 += m[k] * m[k];
    const std::complex<double> det = std::complex<double>(m[0], m[1]) * std::complex<double>(m[6], m[7]) -
                                     std::complex<double>(m[2], m[3]) * std::complex<double>(m[4], m[5]);
    const double d = f2 * f2 - 4.0 * std::norm(det);
    return std::sqrt(0.5 * (f2 + std::sqrt(std::max(d, 0.0))));
}

bool has_block_plan(int n, const llg_op* ops, int nops) {
    if (n < kBlockMinQubits) return false;
    for (int i = 0; i < nops; ++i)
        if (ops[i].kind == LLG_OP_U2 && !(spectral_norm_2x2(ops[i].m) <= kBlockNormLimit)) return false;
    return true;
}

bool keeps_norms(const llg_op* ops, int nops) {
    double drift = 0.0;
    for (int i = 0; i < nops; ++i) {
        if (ops[i].kind != LLG_OP_U2) continue;
        const double* m = ops[i].m;
        // M^+ M = [a, c; conj c, b]: its eigenvalues, the singular values' squares, are this close to 1
        const double a = m[0] * m[0] + m[1] * m[1] + m[4] * m[4] + m[5] * m[5];
        const double b = m[2] * m[2] + m[3] * m[3] + m[6] * m[6] + m[7] * m[7];
        const double cr = m[0] * m[2] + m[1] * m[3] + m[4] * m[6] + m[5] * m[7];
        const double ci = m[0] * m[3] - m[1] * m[2] + m[4] * m[7] - m[5] * m[6];
        const double off = 0.5 * (std::max(std::fabs(a - 1.0), std::fabs(b - 1.0)) + std::fabs(cr) + std::fabs(ci));
        if (!(off <= kBlockNormLimit - 1.0)) return false;
        drift += off;
    }
    return drift <= 0.25;
}

}  // namespace llg
