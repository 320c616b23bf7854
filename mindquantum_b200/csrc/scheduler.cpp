// Host-side pass scheduler.
//
// The reference applies every gate as its own sweep over the state
// (VectorState::ApplyCircuit, ccsrc/include/simulator/vector/vector_state.tpp:949-960).  Here a
// circuit is cut into passes: a fused pass owns a set Q of K "tile" qubits (always including
// the lowest c qubits, so every tile is made of 128-byte contiguous runs) and applies, in one
// read + write of the state, every gate whose non-diagonal targets lie in Q.  Diagonal gates
// and control qubits may sit anywhere: outside Q their bits are constant over a tile.
//
// The greedy scan keeps the circuit's order of gates that share a qubit: a gate that cannot join
// the current pass blocks all its qubits for the rest of the scan, so no later gate sharing a
// qubit with it can overtake it.  The set Q of a pass (and the register bits of a stage) is the one
// of several candidates that takes the most gates (choose_set).
#include <algorithm>
#include <cstdlib>
#include <stdexcept>

#include "mqb_internal.h"

namespace mqb {

static inline int popc(uint64_t x) { return __builtin_popcountll(x); }

int contiguity_bits(int precision) { return precision == MQB_PREC_C64 ? 4 : 3; }

// MQB_FWD_REG_BITS (2..5) overrides the complex64 forward register bits (tuning).
int fwd_reg_bits(int precision) {
    if (precision == MQB_PREC_C64)
        if (const char *e = std::getenv("MQB_FWD_REG_BITS")) return std::max(2, std::min(5, std::atoi(e)));
    return precision == MQB_PREC_C64 ? 5 : 4;
}

int jit_fwd_reg_bits(int precision) { return precision == MQB_PREC_C64 ? std::min(4, fwd_reg_bits(precision)) : fwd_reg_bits(precision); }

int bwd_reg_bits(int precision, int n_hams) {
    if (n_hams <= 1) return precision == MQB_PREC_C64 ? 4 : 3;
    return precision == MQB_PREC_C64 ? 3 : 2;
}

int default_tile_bits(int precision, int n_states_in_tile) {
    // keep the shared-memory tiles of all states at <= 64 KB so 2-3 blocks fit per SM
    const size_t amp = precision == MQB_PREC_C64 ? 8 : 16;
    int K = kMaxTileBits;
    while (K > 6 && (size_t(n_states_in_tile) << K) * amp > 65536) --K;
    return K;
}

TileGeom make_geom(int n, const std::vector<int> &qbits) {
    TileGeom g{};
    g.n = n;
    g.K = int(qbits.size());
    g.c = 0;
    while (g.c < g.K && qbits[g.c] == g.c) ++g.c;
    uint64_t qm = 0;
    for (int i = 0; i < g.K; ++i) {
        g.qbits[i] = int8_t(qbits[i]);
        qm |= uint64_t(1) << qbits[i];
    }
    g.n_out = 0;
    for (int q = 0; q < n; ++q)
        if (!(qm >> q & 1)) g.outside[g.n_out++] = int8_t(q);
    return g;
}

static uint64_t dense_targets(const DevOp &op) {
    if (op.kind != KIND_DENSE) return 0;
    uint64_t m = 0;
    for (int k = 0; k < op.m; ++k) m |= uint64_t(1) << op.tq[k];
    return m;
}

static uint64_t touched(const DevOp &op) {
    uint64_t m = op.ctrl;
    for (int k = 0; k < op.m; ++k) m |= uint64_t(1) << op.tq[k];
    if (op.kind == KIND_RPS) m |= op.px | op.py | op.pz;
    return m;
}

static bool fusable(const DevOp &op) { return (op.kind == KIND_DENSE || op.kind == KIND_DIAG) && op.m <= kMaxFusedM; }

namespace {

// One item of a greedy scan (a gate in build_schedule, a pass op in build_stages): the qubits (bits)
// it touches, the ones that have to be in the chosen set, and what it adds to the limits.
struct ScanItem {
    uint64_t touch = 0, dense = 0;
    int slots = 0, entries = 0;
    bool fusable = true;
    bool apart = false;              // runs only with others of its kind (a non-unitary operator)
};

struct ScanLimits {
    int K = 0;                       // qubits of the set
    int max_items = 1 << 30, max_slots = 1 << 30, max_entries = 1 << 30;
    uint64_t all = 0;
    bool apart = false;              // the kind of items the set is for
    bool boxes = false;              // sets are moved by tensor copies (box_cost)
};

// Time of a pass over the tiles of set Q against one that is moved whole.  A tensor copy takes the low run of consecutive
// qubits and four more; each further run doubles the copies per tile.  Adjoint passes of some 40 gates on 30 qubits: 16.0
// ms with 1 copy per tile, 17.1 with 2, 20.9 with 4, 25.9 with 8 and 39 with 16.
double box_cost(uint64_t Q) {
    static const double cost[] = {1.0, 1.07, 1.3, 1.6, 2.4, 4.0};
    const int runs = popc(Q & ~(Q << 1));
    return cost[std::min(5, std::max(0, runs - 5))];
}

// The items that no group has taken yet, in program order: list[head..).  Removing a group moves the kept items before its last
// one up, so that it costs no more than the scan that found it; the scans, which are many, read an array.
struct Left {
    std::vector<int> list;
    size_t head = 0;

    explicit Left(size_t n) : list(n) {
        for (size_t i = 0; i < n; ++i) list[i] = int(i);
    }
    bool empty() const { return head == list.size(); }
    int front() const { return list[head]; }
    void remove(const std::vector<int> &members) {   // (ascending, not empty)
        size_t from = head, m = members.size();
        while (list[from] != members.back()) ++from;
        size_t to = from + 1;
        for (size_t p = from + 1; p-- > head;) {
            if (m > 0 && list[p] == members[m - 1]) --m;
            else list[--to] = list[p];
        }
        head = to;
    }
};

// The items of `left` that can run together when the set is Q, which
// grows up to K qubits as the items ask for them when `grow`.  An item that cannot join blocks the
// qubits it touches for the rest of the scan.  Returns how many join; `members` may be null; `wanted`
// (optional) gets the qubits outside Q that kept an otherwise free item out.
int scan_items(const std::vector<ScanItem> &items, const Left &left, const ScanLimits &lim, uint64_t &Q,
               bool grow, std::vector<int> *members, uint64_t *wanted = nullptr) {
    uint64_t blocked = 0;
    if (wanted) *wanted = 0;
    int n_items = 0, n_slots = 0, n_entries = 0;
    for (size_t p = left.head; p < left.list.size(); ++p) {
        const int i = left.list[p];
        const ScanItem &it = items[size_t(i)];
        if (n_items >= lim.max_items) break;
        const uint64_t need = it.dense & ~Q;
        if ((it.touch & blocked) || !it.fusable || it.apart != lim.apart || (need && (!grow || popc(Q | need) > lim.K)) ||
            n_slots + it.slots > lim.max_slots || n_entries + it.entries > lim.max_entries) {
            if (wanted && need && !(it.touch & blocked) && it.fusable && it.apart == lim.apart) *wanted |= need;
            blocked |= it.touch;
            if ((blocked & lim.all) == lim.all) break;
            continue;
        }
        Q |= need;
        n_slots += it.slots;
        n_entries += it.entries;
        ++n_items;
        if (members) members->push_back(i);
    }
    return n_items;
}

// The set of at most K qubits, Q0 among them, under which the most items of `left` run together (per time of the pass,
// `lim.boxes`), out of: the qubits in the order the items ask for them; every window of consecutive qubits above
// Q0 (`windows`); and Q0 grown by the qubit that lets most items join, one at a time, freely and (`lim.boxes`) without a
// further run of qubits where that would double the copies per tile.  In a layered circuit a
// set taken in program order is used for about two layers: the gates of later layers wait for
// neighbours outside it.  A window next to the qubits that earlier passes brought furthest lets a
// wedge of many layers through (26 qubits x 12 layers of RY, RZ and a CNOT ladder, 12-qubit sets: 14
// passes instead of 31).  Ties keep the program-order set.
uint64_t choose_set(const std::vector<ScanItem> &items, const Left &left, const ScanLimits &lim,
                    uint64_t Q0, int n, bool windows) {
    uint64_t best_q = Q0;
    const int plain = scan_items(items, left, lim, best_q, true, nullptr);
    if (n <= lim.K) return best_q;
    auto rate = [&](uint64_t Q, int got) { return lim.boxes ? got / box_cost(Q) : double(got); };
    double best = rate(best_q, plain);
    auto offer = [&](uint64_t Q, int got) {
        if (rate(Q, got) > best) {
            best = rate(Q, got);
            best_q = Q;
        }
    };
    const int w = lim.K - popc(Q0);
    if (windows && w > 0 && w < 64) {
        const int low = popc(Q0);
        for (int a = low; a + w <= n; ++a) {
            uint64_t Q = Q0 | (((uint64_t(1) << w) - 1) << a);
            if (popc(Q) == lim.K) offer(Q, scan_items(items, left, lim, Q, false, nullptr));
        }
    }
    for (int whole = 0; whole <= (lim.boxes ? 1 : 0); ++whole) {
        uint64_t Q = Q0, wanted = 0;
        int got = scan_items(items, left, lim, Q, false, nullptr, &wanted);
        bool met = false;   // the second growth differs from the first
        while (popc(Q) < lim.K && wanted) {   // only a wanted qubit lets more items join
            int step_got = -1;
            uint64_t step_q = Q, step_wanted = 0;
            for (uint64_t rest = wanted; rest; rest &= rest - 1) {
                uint64_t t = Q | (rest & ~(rest - 1)), w = 0;
                if (whole && box_cost(t) > box_cost(Q)) {
                    met = true;
                    continue;
                }
                const int g = scan_items(items, left, lim, t, false, nullptr, &w);
                if (g > step_got) {
                    step_got = g;
                    step_q = t;
                    step_wanted = w;
                }
            }
            if (step_got < 0) break;
            Q = step_q;
            got = step_got;
            wanted = step_wanted;
        }
        if (!whole || met) offer(Q, got);
        if (!whole && box_cost(Q) == 1.0) break;
    }
    return best_q;
}

// A group of items that run together under one set; `single`: an item that runs alone, outside any set.
struct Cut {
    uint64_t set = 0;
    std::vector<int> members;
    bool single = false;
};

// Cut the items into groups, each group's set taken in program order or, with `search`, by choose_set.
std::vector<Cut> cut_items(const std::vector<ScanItem> &items, ScanLimits lim, uint64_t Q0, int n, bool windows,
                           bool search) {
    Left left(items.size());
    std::vector<Cut> out;
    while (!left.empty()) {
        Cut c;
        if (items[size_t(left.front())].fusable) {
            c.set = Q0;
            lim.apart = items[size_t(left.front())].apart;
            if (search) c.set = choose_set(items, left, lim, Q0, n, windows);
            scan_items(items, left, lim, c.set, !search, &c.members);
        }
        if (c.members.empty()) {
            // not fusable, or too wide for the room next to Q0
            c.single = true;
            c.members.push_back(left.front());
        }
        left.remove(c.members);
        out.push_back(std::move(c));
    }
    return out;
}

// The cut with fewer groups (`lim.boxes`: of less time); program order where the search saves none (its groups are more even).
std::vector<Cut> best_cut(const std::vector<ScanItem> &items, const ScanLimits &lim, uint64_t Q0, int n, bool windows,
                          bool search) {
    std::vector<Cut> plain = cut_items(items, lim, Q0, n, windows, false);
    if (!search || n <= lim.K || plain.size() < 3) return plain;
    std::vector<Cut> found = cut_items(items, lim, Q0, n, windows, true);
    auto time = [&](const std::vector<Cut> &cuts) {
        double t = 0;
        for (const Cut &c : cuts) t += lim.boxes ? box_cost(c.set) : 1.0;
        return t;
    };
    return time(found) < time(plain) ? found : plain;
}

}  // namespace

Schedule build_schedule(int n, int K, int c, const std::vector<DevOp> &ops, bool fuse, const std::vector<char> *apart,
                        const PassLimits &limits) {
    Schedule s;
    if (K > n) K = n;
    // leave room for the widest fused gate next to the contiguity bits; keep at least one
    // contiguity bit so 16-byte vector accesses never straddle two tile runs
    if (c > K - kMaxFusedM) c = std::max(1, K - kMaxFusedM);
    if (n > K && K < kMaxFusedM + 1) fuse = false;
    if (K < 6) fuse = false;
    s.K = K;
    s.search = limits.search;
    const int L = int(ops.size());
    const uint64_t all = n >= 64 ? ~uint64_t(0) : ((uint64_t(1) << n) - 1);
    std::vector<ScanItem> items(static_cast<size_t>(L));
    for (int i = 0; i < L; ++i) {
        ScanItem &it = items[size_t(i)];
        it.touch = touched(ops[i]);
        it.dense = dense_targets(ops[i]);
        it.slots = popc(uint64_t(ops[i].grad_mask));
        it.entries = ops[i].mat_size * (1 + (limits.derivatives && ops[i].grad_mask ? ops[i].n_angles : 0));
        it.fusable = fuse && fusable(ops[i]);
        it.apart = apart && (*apart)[i];
    }
    ScanLimits lim;
    lim.K = K;
    lim.max_items = kMaxPassOps;
    lim.max_slots = kMaxPassSlots;
    lim.max_entries = limits.max_entries;
    lim.boxes = limits.boxes;
    for (const ScanItem &it : items) lim.all |= it.touch;   // (a scan ends when they are blocked: idle qubits never are)
    for (const Cut &cut : best_cut(items, lim, (n <= K) ? all : ((uint64_t(1) << c) - 1), n, true, limits.search)) {
        const std::vector<int> &members = cut.members;
        if (cut.single) {
            const int first = members.front();
            Pass p;
            p.fused = 0;
            p.op_begin = first;
            p.op_end = first + 1;
            p.prog_op_begin = first;
            p.prog_op_end = first + 1;
            s.passes.push_back(p);
            continue;
        }
        uint64_t Q = cut.set;
        // pad the tile to exactly K qubits with the lowest free qubits
        for (int q = 0; q < n && popc(Q) < K; ++q) Q |= uint64_t(1) << q;
        Pass p;
        p.fused = 1;
        p.K = K;
        for (int q = 0; q < n; ++q) {
            if (Q >> q & 1)
                p.qbits.push_back(q);
            else
                p.outside.push_back(q);
        }
        p.c = 0;
        while (p.c < K && p.qbits[p.c] == p.c) ++p.c;
        int local[64];
        for (int i = 0; i < 64; ++i) local[i] = -1;
        for (int i = 0; i < K; ++i) local[p.qbits[i]] = i;
        p.op_begin = int(s.pass_ops.size());
        p.slot_begin = int(s.slot_map.size());
        for (int i : members) {
            const DevOp &op = ops[i];
            PassOp po{};
            po.op = i;
            po.kind = op.kind;
            po.m = op.m;
            for (int k = 0; k < kMaxFusedM; ++k) {
                po.lt[k] = -1;
                po.gt[k] = 0;
            }
            for (int k = 0; k < op.m; ++k) {
                po.gt[k] = op.tq[k];
                po.lt[k] = local[op.tq[k]];
                if (op.kind == KIND_DENSE && po.lt[k] < 0) throw std::logic_error("dense target outside tile");
            }
            po.lctrl = 0;
            po.octrl = 0;
            for (int q = 0; q < n; ++q) {
                if (!(op.ctrl >> q & 1)) continue;
                if (local[q] >= 0)
                    po.lctrl |= 1u << local[q];
                else
                    po.octrl |= uint64_t(1) << q;
            }
            po.lslot = -1;
            if (op.grad_mask) {
                po.lslot = int(s.slot_map.size()) - p.slot_begin;
                for (int a = 0, r = 0; a < op.n_angles; ++a)
                    if (op.grad_mask >> a & 1) s.slot_map.push_back(op.slot0 + r++);
            }
            s.pass_ops.push_back(po);
        }
        p.op_end = int(s.pass_ops.size());
        p.n_slots = int(s.slot_map.size()) - p.slot_begin;
        p.prog_op_begin = members.front();
        p.prog_op_end = members.back() + 1;
        s.passes.push_back(p);
    }
    return s;
}

// Greedy register-stage grouping of one fused pass (same blocking rule as the pass scan, over
// tile-local bits), then padding of the register set and a bank-conflict-aware thread-bit order.
// Register code (forward) and code * 4 + gradient selector (backward) of a stage op; ops whose
// shape or gradient angles have no specialised kernel take the generic codes.
void assign_codes(StageOp &so) {
    const int nrc = popc(so.rctrl);
    const int C = nrc == 1 ? __builtin_ctz(so.rctrl) : -1;
    const int gm = so.n_angles ? so.grad_mask : 0;
    int code = -1, gsel = 0;
    switch (so.kind) {
        case SK_DENSE1:
        case SK_REAL1:
        case SK_RXL1:
        case SK_PERM1:
        case SK_SWAP1: {
            const int P = so.p0;
            if (nrc == 0) {
                if (so.kind == SK_SWAP1) code = RC_X1 + P;
                else if (so.kind == SK_REAL1) code = RC_REAL1 + P;
                else if (so.kind == SK_RXL1) code = RC_RXL1 + P;
                else code = RC_DENSE1 + P;
            } else if (nrc == 1) {
                code = so.kind == SK_SWAP1 ? RC_X1C + 5 * P + C : RC_DENSE1C + 5 * P + C;
            } else {
                code = RC_GDENSE1 + P;
            }
            // gradient selector; what the specialised kernels lack goes generic
            const bool x = code >= RC_X1 && code < RC_X1 + 5;
            const bool xc = code >= RC_X1C && code < RC_X1C + 25;
            if (gm == 0) {
                gsel = code >= RC_GDENSE1 ? 3 : 0;
            } else if ((x || xc) && gm) {
                code = RC_GDENSE1 + P;   // X matrices carry no derivative; never reached by lowered gates
                gsel = 3;
            } else if (code >= RC_GDENSE1) {
                gsel = 3;
            } else if (gm == 1) {
                gsel = 1;
            } else if (code < RC_DENSE1 + 5 && gm == 7) {
                gsel = 2;
            } else if (code < RC_DENSE1 + 5) {
                gsel = 3;
            } else {
                code = RC_GDENSE1 + P;
                gsel = 3;
            }
        } break;
        case SK_DENSE2: {
            const int P = so.p0, Q = so.p1;
            if (nrc == 0) {
                code = RC_DENSE2 + 5 * P + Q;
                gsel = gm == 0 ? 0 : gm == 1 ? 1 : 3;
            } else {
                code = RC_GDENSE2 + 5 * P + Q;
                gsel = 3;
            }
        } break;
        case SK_DIAG1:
        case SK_DIAG2: {
            const bool two = so.kind == SK_DIAG2;
            const bool in0 = so.dsrc[0] == 0, in1 = two && so.dsrc[1] == 0;
            if (gm != 0 && gm != 1) {
                code = RC_GDIAG;
            } else if (!two) {
                if (in0) code = nrc == 0 ? RC_DIAG1 + so.dval[0] : nrc == 1 ? RC_DIAG1C + 5 * so.dval[0] + C : RC_GDIAG;
                else code = nrc == 0 ? RC_SCALE : nrc == 1 ? RC_SCALEC + C : RC_GDIAG;
            } else if (nrc != 0) {
                code = RC_GDIAG;
            } else if (in0 && in1) {
                code = RC_DIAG2 + 5 * so.dval[0] + so.dval[1];
            } else if (in0) {
                code = RC_DIAG2S + so.dval[0];
            } else if (in1) {
                code = RC_DIAG2S + 5 + so.dval[1];
            } else {
                code = RC_SCALE;
            }
            gsel = code == RC_GDIAG ? 3 : gm;
        } break;
        default:
            throw std::runtime_error("stage op of unknown kind");
    }
    so.code = code;
    so.bcode = code * 4 + gsel;
    so.cflags = (so.octrl ? 1 : 0) | (so.tctrl ? 2 : 0);
}

void build_stages(Schedule &s, const std::vector<DevOp> &ops, int reg_bits, int precision, bool forward) {
    std::vector<StageDesc> &stages = forward ? s.f_stages : s.stages;
    std::vector<StageOp> &stage_ops = forward ? s.f_stage_ops : s.stage_ops;
    stages.clear();
    stage_ops.clear();
    const int res_mod = precision == MQB_PREC_C64 ? 4 : 3;
    for (Pass &p : s.passes) {
        if (!p.fused) continue;
        const int K = p.K;
        // 2^TB threads (32..256) holding 2^RB amplitudes each; passes are only fused when K >= reg_bits + 5
        const int RB = std::min(reg_bits, K - 5);
        const int TB = K - RB;
        const int stage_begin = int(stages.size());
        const int sop_begin = int(stage_ops.size());
        int mtab = 0;
        const int npo = p.op_end - p.op_begin;
        std::vector<ScanItem> items(static_cast<size_t>(npo));
        for (int i = 0; i < npo; ++i) {
            const PassOp &po = s.pass_ops[p.op_begin + i];
            ScanItem &it = items[size_t(i)];
            it.touch = po.lctrl;
            for (int k = 0; k < po.m; ++k)
                if (po.lt[k] >= 0) it.touch |= 1u << po.lt[k];
            if (po.kind == KIND_DENSE) it.dense = it.touch & ~uint64_t(po.lctrl);
        }
        ScanLimits lim;
        lim.K = RB;
        lim.all = (uint64_t(1) << K) - 1;
        for (const Cut &cut : best_cut(items, lim, 0, K, false, s.search)) {
            const std::vector<int> &members = cut.members;
            // keep only the bits that a member needs: the rest is padded below
            uint32_t R = 0;
            for (int i : members) R |= uint32_t(items[size_t(i)].dense);
            // padding: add local bits so that the thread bits keep one bit of every residue class
            auto thread_residue_count = [&](uint32_t Rm, int r) {
                int cnt = 0;
                for (int b = 0; b < K; ++b)
                    if (!(Rm >> b & 1) && b % res_mod == r) ++cnt;
                return cnt;
            };
            // (ties go to the highest bit: the low contiguous bits stay thread bits, so a stage can
            // read and write the tile in the order the TMA lands it without bank conflicts)
            while (popc(R) < RB) {
                int best = -1, best_score = -1;
                for (int b = K - 1; b >= 0; --b) {
                    if (R >> b & 1) continue;
                    const int score = thread_residue_count(R, b % res_mod);
                    if (score > best_score) {
                        best_score = score;
                        best = b;
                    }
                }
                R |= 1u << best;
            }
            StageDesc sd{};
            std::vector<int> rl;
            for (int b = 0; b < K; ++b)
                if (R >> b & 1) rl.push_back(b);
            // register positions: dense targets first in op order are not needed; ascending is fine
            for (int i = 0; i < RB; ++i) sd.rbits[i] = int8_t(rl[i]);
            std::vector<int> tl;
            for (int b = 0; b < K; ++b)
                if (!(R >> b & 1)) tl.push_back(b);
            // lanes first: one thread bit of each residue class, then the rest ascending
            std::vector<int> order;
            std::vector<char> used(tl.size(), 0);
            for (int r = 0; r < res_mod; ++r)
                for (size_t i = 0; i < tl.size(); ++i)
                    if (!used[i] && tl[i] % res_mod == r) {
                        order.push_back(tl[i]);
                        used[i] = 1;
                        break;
                    }
            for (size_t i = 0; i < tl.size(); ++i)
                if (!used[i]) order.push_back(tl[i]);
            for (int i = 0; i < TB; ++i) sd.tbits[i] = int8_t(order[i]);
            int pos_of[32];
            for (int i = 0; i < 32; ++i) pos_of[i] = -1;
            for (int i = 0; i < RB; ++i) pos_of[rl[i]] = i;
            sd.op_begin = int(stage_ops.size()) - sop_begin;
            for (int i : members) {
                const PassOp &po = s.pass_ops[p.op_begin + i];
                const DevOp &dop = ops[po.op];
                StageOp so{};
                so.op = po.op;
                so.lslot = po.lslot;
                so.grad_mask = dop.grad_mask;
                so.n_angles = dop.grad_mask ? dop.n_angles : 0;
                so.mat_size = dop.mat_size;
                so.moff = mtab;
                so.mcount = forward ? dop.mat_size : dop.mat_size * (1 + so.n_angles);   // a forward pass reads M alone
                so.msrc = dop.mat_off;
                so.msrc_ps = dop.per_sample;
                mtab += so.mcount;
                so.octrl = po.octrl;
                so.rctrl = 0;
                so.tctrl = 0;
                for (int b = 0; b < K; ++b) {
                    if (!(po.lctrl >> b & 1)) continue;
                    if (pos_of[b] >= 0)
                        so.rctrl |= 1u << pos_of[b];
                    else
                        so.tctrl |= 1u << b;
                }
                if (po.kind == KIND_DENSE) {
                    so.kind = po.m == 1 ? SK_DENSE1 : SK_DENSE2;
                    if (po.m == 1 && dop.sub == SUB_REAL) so.kind = SK_REAL1;
                    if (po.m == 1 && dop.sub == SUB_PERM) so.kind = SK_PERM1;
                    if (po.m == 1 && dop.sub == SUB_SWAP) so.kind = SK_SWAP1;
                    if (po.m == 1 && dop.sub == SUB_RXL) so.kind = SK_RXL1;
                    so.p0 = pos_of[po.lt[0]];
                    so.p1 = po.m == 2 ? pos_of[po.lt[1]] : 0;
                } else {
                    so.kind = po.m == 1 ? SK_DIAG1 : SK_DIAG2;
                    so.dsrc[1] = 3;   // absent second target
                    so.dval[1] = 0;
                    for (int k = 0; k < po.m; ++k) {
                        if (po.lt[k] >= 0 && pos_of[po.lt[k]] >= 0) {
                            so.dsrc[k] = 0;
                            so.dval[k] = pos_of[po.lt[k]];
                        } else if (po.lt[k] >= 0) {
                            so.dsrc[k] = 1;
                            so.dval[k] = po.lt[k];
                        } else {
                            so.dsrc[k] = 2;
                            so.dval[k] = po.gt[k];
                        }
                    }
                }
                assign_codes(so);
                so.unitary = dop.unitary != 0;
                // the norm that rounding gave an uncontrolled complex64 gate is measured (of the constant matrices only the
                // first gate's on a qubit: on the structured states of Clifford circuits the later ones cancel)
                if (precision == MQB_PREC_C64 && !dop.ctrl && so.kind != SK_SWAP1 && (dop.unitary == 2 || (dop.unitary && dop.per_sample)))
                    so.norm = int16_t(so.kind == SK_DIAG1 ? -2 : so.kind == SK_DIAG2 ? -4 : so.kind == SK_DENSE2 ? 4 : 2);
                stage_ops.push_back(so);
            }
            sd.op_end = int(stage_ops.size()) - sop_begin;
            stages.push_back(sd);
        }
        std::vector<const StageDesc *> order;   // of execution
        for (size_t k = size_t(stage_begin); k < stages.size(); ++k) order.push_back(&stages[k]);
        if (!forward) std::reverse(order.begin(), order.end());
        (forward ? p.f_run_entries : p.run_entries) = jit_run_entries(order, stage_ops.data() + sop_begin, ops, precision, !forward);
        if (forward) {
            p.f_reg_bits = RB;
            p.f_stage_begin = stage_begin;
            p.f_n_stages = int(stages.size()) - stage_begin;
            p.f_sop_begin = sop_begin;
            p.f_n_sops = int(stage_ops.size()) - sop_begin;
            p.f_mtab_entries = mtab;
        } else {
            p.reg_bits = RB;
            p.thread_bits = TB;
            p.stage_begin = stage_begin;
            p.n_stages = int(stages.size()) - stage_begin;
            p.sop_begin = sop_begin;
            p.n_sops = int(stage_ops.size()) - sop_begin;
            p.mtab_entries = mtab;
        }
    }
}

void build_ham_groups(int n, int K, int c, const std::vector<uint64_t> &mx, const std::vector<uint64_t> &my,
                      const std::vector<uint64_t> &mz, const std::vector<int> &ny, const std::vector<double> &coeff,
                      std::vector<HamGroup> &groups, std::vector<HamClass> &classes, std::vector<HamTerm> &terms) {
    if (K > n) K = n;
    if (c > K) c = K;
    const int T = int(coeff.size());
    // classes: distinct flip masks, in order of first appearance
    std::vector<uint64_t> flips;
    std::vector<std::vector<int>> members;
    for (int t = 0; t < T; ++t) {
        const uint64_t f = mx[t] | my[t];
        auto it = std::find(flips.begin(), flips.end(), f);
        if (it == flips.end()) {
            flips.push_back(f);
            members.push_back({t});
        } else {
            members[it - flips.begin()].push_back(t);
        }
    }
    // split oversized classes
    std::vector<uint64_t> cflip;
    std::vector<std::vector<int>> cmem;
    for (size_t i = 0; i < flips.size(); ++i) {
        for (size_t s = 0; s < members[i].size(); s += kMaxClassTerms) {
            cflip.push_back(flips[i]);
            cmem.emplace_back(members[i].begin() + s,
                              members[i].begin() + std::min(members[i].size(), s + size_t(kMaxClassTerms)));
        }
    }
    const uint64_t all = n >= 64 ? ~uint64_t(0) : ((uint64_t(1) << n) - 1);
    std::vector<char> used(cflip.size(), 0);
    size_t n_used = 0;
    while (n_used < cflip.size()) {
        uint64_t Q = (n <= K) ? all : ((uint64_t(1) << c) - 1);
        std::vector<int> in_group;
        for (size_t i = 0; i < cflip.size() && int(in_group.size()) < kMaxGroupClasses; ++i) {
            if (used[i]) continue;
            if (popc(Q | cflip[i]) <= K) {
                Q |= cflip[i];
                in_group.push_back(int(i));
                used[i] = 1;
                ++n_used;
            }
        }
        if (in_group.empty()) throw std::runtime_error("Pauli term acts on more qubits than a tile holds");
        for (int q = 0; q < n && popc(Q) < K; ++q) Q |= uint64_t(1) << q;
        std::vector<int> qb;
        for (int q = 0; q < n; ++q)
            if (Q >> q & 1) qb.push_back(q);
        HamGroup g{};
        g.geom = make_geom(n, qb);
        g.class_begin = int(classes.size());
        g.class_count = int(in_group.size());
        for (int ci : in_group) {
            HamClass hc{};
            hc.flip = cflip[ci];
            hc.lflip = 0;
            for (int i = 0; i < g.geom.K; ++i)
                if (hc.flip >> g.geom.qbits[i] & 1) hc.lflip |= 1u << i;
            hc.term_begin = int(terms.size());
            hc.term_count = int(cmem[ci].size());
            const int K = g.geom.K;
            const int shift = std::max(0, K - kHamRegBits);
            std::vector<HamTerm> ts;
            for (int t : cmem[ci]) {
                HamTerm ht{};
                ht.coeff = coeff[t];
                ht.my_mz = my[t] | mz[t];
                ht.ny = ny[t];
                ht.lmask = 0;
                for (int i = 0; i < K; ++i)
                    if (ht.my_mz >> g.geom.qbits[i] & 1) ht.lmask |= 1u << i;
                uint64_t tile_q = 0;
                for (int i = 0; i < K; ++i) tile_q |= uint64_t(1) << g.geom.qbits[i];
                ht.omask = ht.my_mz & ~tile_q;
                // i^ny (ny counts the Y factors, each Y contributing i) and the flip's sign
                const int ph = (ny[t] + 2 * popc(hc.flip & ht.my_mz)) & 3;
                ht.cb_re = ph == 0 ? coeff[t] : ph == 2 ? -coeff[t] : 0.0;
                ht.cb_im = ph == 1 ? coeff[t] : ph == 3 ? -coeff[t] : 0.0;
                ts.push_back(ht);
            }
            auto bin_of = [&](const HamTerm &ht) { return int((ht.lmask >> shift) & ((1u << kHamRegBits) - 1)); };
            std::stable_sort(ts.begin(), ts.end(), [&](const HamTerm &x, const HamTerm &y) { return bin_of(x) < bin_of(y); });
            for (int b = 0, q = 0; b <= (1 << kHamRegBits); ++b) {
                while (q < int(ts.size()) && bin_of(ts[q]) < b) ++q;
                hc.bins[b] = q;
            }
            terms.insert(terms.end(), ts.begin(), ts.end());
            classes.push_back(hc);
        }
        groups.push_back(g);
    }
}

}  // namespace mqb
