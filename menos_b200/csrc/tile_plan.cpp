// Host planner of the multi-gate tiled sweep.
//
// A pass loads every tile of 2^m amplitudes -- the amplitudes that share
// their bits outside a set S of m qubits -- into shared memory once, applies
// a run of blocks whose operands lie in S, and writes the tile back once.
// A pass applies blocks in their order (exact ones may move past blocks on
// other qubits), and per amplitude the arithmetic of every block is exactly
// the per-gate kernel's, so the state after the sweep is bitwise the one the reference's
// block-by-block sweep gives
// (src/engines/dense/fused_block.h:60-101, src/engines/dense/dense_engine.cpp:65-112).
//
// Inside a pass each thread holds 16 amplitudes in registers (4 "register
// qubits"); a PHASE instruction picks which 4 tile qubits those are, and the
// blocks of the phase act on registers only.  Diagonal blocks need no pairing
// and run in any phase.  Blocks wider than 2 dense qubits run from shared
// memory (TOP_SMEM).
#include <algorithm>
#include <bit>
#include <cmath>
#include <initializer_list>
#include <stdexcept>

#include "mb2_internal.h"

namespace mb2 {
namespace {

constexpr size_t kMaxBlocksPerPass = 300;

// How far behind a closed pass exact moves are looked for that may still run
// in it.  Usually the blocks held back soon cover every qubit; they never do
// where a qubit has no blocks, or has them only far behind.  Looking through
// the whole rest of the program for each pass, 1000 brick layers on 19 of 20
// qubits took 409 ms to plan (66 before moves were looked for, 54 now).  512
// blocks are six layers of a 28-qubit RY/RZ + CX ansatz, whose plans it leaves
// as they are.
constexpr size_t kMaxAhead = 512;

// States up to which a program's passes run one kernel (TilePass::mapped): one
// and two kernels, ms: a sampled density matrix of 10 and 11 qubits (20 and 22
// here; its passes are of both kinds) 0.601 0.634, 1.184 1.208; 10 brick layers
// and a CX ladder at 20 qubits 0.316 0.318, at 22 1.039 1.049, at 23 2.115
// 2.110, at 24 4.46 4.43; 5 layers at 26 10.48 10.28.
constexpr uint32_t kOneKernelQubits = 22;

// A pass's instruction words and small-matrix data are staged in shared memory
// (kMaxStagedBytes): a bound on what each block adds, whatever order the
// pass's blocks come in.
//
// Phase records: a dense block of one or two qubits opens at most one.  A
// diagonal runs in whatever phase is open, so it opens one only at the pass's
// start (base), behind a permutation or behind a wide block (k >= 3), and is
// held by those: a permutation counts one record, a wide block one, and in a
// program with permutations one more, for the phase that brings moved
// amplitudes back before it.  Every record is counted as large as a program
// with permutations may need it.
// Words beside them: a gate's, at most one extra and its phase's end for a
// dense block or a diagonal, a wide block's three and the end of the phase
// that brings amplitudes back.
struct Staged {
    uint32_t m;
    bool mapped, c64;  // the program has permutations; it is the complex64 kernels'
    bool tc = false;   // every pass is rewritten for the tensor cores
    size_t operator()(const Block& b, bool move) const {
        const size_t dim = size_t{1} << b.k;
        // Nothing of this is staged then; 128 bytes a block and its entries
        // make passes whose phase matrices fill the room they have (longer ones
        // are split and leave short ends: 17 passes instead of 14 for the
        // unfused 30-qubit ansatz of 10 layers).
        if (tc) return 128 + (b.diagonal ? dim : dim * dim) * 2 * sizeof(double);
        const bool wide = !b.diagonal && b.k > 2;
        const size_t entries = move || wide ? 0 : b.diagonal ? dim : dim * dim;
        const size_t record = mapped ? cop::phase_map_words(m) + (c64 ? 0 : cop::kMaxMapControls) : cop::phase_words(m);
        const size_t records = b.diagonal ? 0 : wide && mapped ? 2 : 1;
        return (records * record + (move ? 0 : wide ? 4 : 3)) * sizeof(uint32_t) + entries * 2 * sizeof(double);
    }
    size_t base() const { return tc ? 0 : cop::phase_map_words(m) * sizeof(uint32_t); }
};

uint32_t local_pos(uint64_t smask, uint32_t q) {
    return static_cast<uint32_t>(std::popcount(smask & ((uint64_t{1} << q) - 1)));
}

bool is_real(const Cd& c) { return c.imag() == 0.0; }
bool is_zero(const Cd& c) { return c.real() == 0.0 && c.imag() == 0.0; }

// Row r's single nonzero column, -1 for an all-zero row, -2 if the row has more.
int mono_src(const std::vector<Cd>& m, uint32_t dim, uint32_t r) {
    int src = -1;
    for (uint32_t c = 0; c < dim; ++c) {
        if (!is_zero(m[r * dim + c])) {
            if (src != -1) return -2;
            src = static_cast<int>(c);
        }
    }
    return src;
}

// The exact permutations that a TileMap takes (X, SWAP, CX either way round),
// or -1.
int move_kind(const Block& b) {
    if (b.diagonal || b.k > 2) return -1;
    const uint32_t dim = 1u << b.k;
    uint32_t rows = 0;
    for (uint32_t r = 0; r < dim; ++r) {
        const int c = mono_src(b.m, dim, r);
        if (c < 0 || b.m[r * dim + static_cast<uint32_t>(c)] != Cd(1.0, 0.0)) return -1;
        rows |= static_cast<uint32_t>(c) << (4 * r);
    }
    if (b.k == 1) return rows == 0x01u ? TK_X : -1;
    return rows == 0x3120u ? TK_SW12 : rows == 0x1230u ? TK_SW13 : rows == 0x2310u ? TK_SW23 : -1;
}

// A two-qubit block that is an exact permutation and a one-qubit gate, in one
// order or the other (a rotation fused with the CX before it, the commonest
// block of an RY/RZ + CX ansatz): split into the two.  Every row of the block
// has the gate's two entries and zeros, a zero entry's product changes at most
// the sign of a zero, and the sum of two products does not depend on their
// order, so the two give the block's bits -- with 12 or 14 FP64 operations per
// amplitude instead of 30, and the permutation taken by the tile's map.
// first, second: the parts in application order.
bool split_block(const Block& b, Block& first, Block& second) {
    if (b.k != 2 || b.diagonal) return false;
    static constexpr uint32_t kPerms[4][4] = {{0, 1, 2, 3}, {0, 2, 1, 3}, {0, 3, 2, 1}, {0, 1, 3, 2}};
    for (uint32_t r = 0; r < 4; ++r) {  // at most two entries a row
        uint32_t entries = 0;
        for (uint32_t c = 0; c < 4; ++c) entries += is_zero(b.m[4 * r + c]) ? 0u : 1u;
        if (entries > 2) return false;
    }
    for (const auto& p : kPerms)
        for (uint32_t t = 0; t < 2; ++t)
            for (const bool gate_last : {true, false}) {
                // gate_last: m[o][i] = u[o][p(i)]; else u[p(o)][i], u on operand t.
                auto at = [&](uint32_t o, uint32_t i) { return gate_last ? b.m[4 * o + p[i]] : b.m[4 * p[o] + i]; };
                const uint32_t bit = 1u << t;
                const Cd u[4] = {at(0, 0), at(0, bit), at(bit, 0), at(bit, bit)};
                bool same = true;
                for (uint32_t o = 0; o < 4 && same; ++o)
                    for (uint32_t i = 0; i < 4 && same; ++i)
                        same = at(o, i) == (((o ^ i) & ~bit) ? Cd(0.0, 0.0) : u[2 * ((o >> t) & 1u) + ((i >> t) & 1u)]);
                if (!same) continue;
                Block perm, gate;
                perm.k = 2;
                perm.q[0] = b.q[0];
                perm.q[1] = b.q[1];
                perm.m.assign(16, Cd(0.0, 0.0));
                for (uint32_t o = 0; o < 4; ++o) perm.m[4 * o + p[o]] = Cd(1.0, 0.0);
                perm.diagonal = p[1] == 1 && p[2] == 2;
                gate.k = 1;
                gate.q[0] = b.q[t];
                gate.m.assign(u, u + 4);
                gate.diagonal = mb2::is_diagonal(gate.m, 2);
                first = gate_last ? std::move(perm) : std::move(gate);
                second = gate_last ? std::move(gate) : std::move(perm);
                return true;
            }
    return false;
}

// A real two-qubit block whose entries lie on the two diagonals: it pairs
// local index 0 with 3 and 1 with 2.  The superoperators of the common
// channels (depolarizing, damping, flips) on a qubit's row and column bits
// are such blocks.
bool is_cross(const Block& b) {
    if (b.k != 2) return false;
    for (uint32_t r = 0; r < 4; ++r)
        for (uint32_t c = 0; c < 4; ++c) {
            const Cd& v = b.m[4 * r + c];
            if (!is_real(v) || (!is_zero(v) && c != r && c != 3 - r)) return false;
        }
    return true;
}

struct PassSel {
    uint64_t smask;
    uint64_t gmask = 0;           // qubits outside the tile that diagonals of the pass read
    std::vector<uint32_t> gates;  // block indices in application order
};

// A diagonal block's operands need not lie in the tile: an amplitude's entry
// depends only on its operand bits, and a qubit outside the tile has one
// value over the whole tile, which the kernel reads off the tile's base
// index.  That holds for the instructions that take an operand as a bit
// value -- diagonals of at most two operands and +-1 diagonals (sign
// monomials) -- not for the wide entry-index diagonal (kDiagK).
bool diagonal_any_operand(const Block& b, bool parametric) {
    if (!b.diagonal) return false;
    if (b.k <= 2) return true;
    if (parametric) return false;
    const uint32_t dim = 1u << b.k;
    for (uint32_t e = 0; e < dim; ++e) {
        const Cd& d = b.m[size_t{e} * dim + e];
        if (d.imag() != 0.0 || (d.real() != 1.0 && d.real() != -1.0)) return false;
    }
    return true;
}

// A diagonal operand's instruction position: its tile position, or
// kGlobalPos0 + its rank among the pass's outside qubits.
uint32_t operand_pos(uint64_t smask, uint64_t gmask, uint32_t q) {
    if ((smask >> q) & 1u) return local_pos(smask, q);
    if (!((gmask >> q) & 1u)) throw std::logic_error("diagonal operand neither in the tile nor global");
    return kGlobalPos0 + static_cast<uint32_t>(std::popcount(gmask & ((uint64_t{1} << q) - 1)));
}

// A block that moves amplitudes and multiplies them by 1, -1, i or -i (X, Y,
// CX, CCX): no output is rounded.  (SWAP too, but the SWAPs that close a QFT
// wait for the qubits that are held back: moving them saves no pass.)
bool is_exact_move(const Block& b) {
    if (b.diagonal || move_kind(b) == TK_SW12) return false;
    const uint32_t dim = 1u << b.k;
    for (uint32_t r = 0; r < dim; ++r) {
        const int c = mono_src(b.m, dim, r);
        if (c < 0) return false;
        const Cd& v = b.m[r * dim + static_cast<uint32_t>(c)];
        if (std::abs(v.real()) + std::abs(v.imag()) != 1.0 || (v.real() != 0.0 && v.imag() != 0.0)) return false;
    }
    return true;
}

// Passes of the plain path, bitwise the reference's sweep, which applies the
// blocks in plan order.  Two gates on disjoint qubits applied in the other
// order give the same state only up to rounding, so a pass takes the blocks as
// they come until one does not fit its tile (diagonals read up to
// kMaxGlobalQubits qubits outside it), and blocks that round never change
// places.  An exact move is another matter.  It changes which amplitudes a
// block on other qubits pairs with which, and their signs or parts (times
// +-i) alike for all the amplitudes of a pair, and rounding is symmetric in
// signs and parts: the two give the same bits in either order.  So behind the
// block that closed the pass, exact moves still run in it when they share no
// qubit with it nor with any block held back since.  A CX ladder then follows
// the layer of rotations it belongs to tile by tile instead of in passes of
// its own: the 16-qubit RY/RZ + CX ansatz of 8 layers takes 13 passes
// instead of 28 (a CX's control, one bit for a whole tile when it lies
// outside, need not be in it either).
std::vector<PassSel> select_passes(const std::vector<Block>& blocks, uint32_t n, uint32_t m, uint32_t fixed_low,
                                   const std::vector<uint8_t>* parametric, const std::vector<int8_t>& kinds) {
    std::vector<PassSel> passes;
    uint32_t widest = 1;
    for (const Block& b : blocks) widest = std::max(widest, b.k);
    const uint32_t mt = std::min(m, n);
    if (widest > mt) throw std::invalid_argument("a block is wider than the tile");
    // Low qubits kept in every tile so that tiles gather contiguous runs,
    // leaving room for the widest block.
    const uint32_t fixed = std::min(fixed_low, mt - widest);
    // Qubits outside the tile that the diagonals read, once the tile is
    // padded to mt qubits with them first.
    auto outside = [&](uint64_t s, uint64_t d) {
        return std::popcount(d & ~s) - (static_cast<int>(mt) - std::popcount(s));
    };
    const size_t nb = blocks.size();
    auto is_param = [&](size_t i) { return parametric != nullptr && ((*parametric)[i] & kParamBlock) != 0; };
    std::vector<uint8_t> moves(nb), done(nb, 0);
    bool mapped = false, any = false;
    for (size_t i = 0; i < nb; ++i) {
        moves[i] = !is_param(i) && is_exact_move(blocks[i]);
        any = any || moves[i];
        mapped = mapped || kinds[i] >= 0;
    }
    std::vector<uint64_t> moves_from(nb + 1, 0);  // qubits of the exact moves from block i on
    for (size_t i = any ? nb : 0; i-- > 0;) moves_from[i] = moves_from[i + 1] | (moves[i] ? blocks[i].mask() : 0);
    const Staged staged_of{mt, mapped, false};
    for (size_t first = 0; first < nb;) {
        uint64_t smask = 0, dmask = 0;  // the tile's qubits so far; the diagonals' operands
        for (uint32_t q = 0; q < fixed; ++q) smask |= uint64_t{1} << q;
        PassSel sel;
        size_t staged = staged_of.base();
        uint64_t held = 0;  // qubits of the blocks held back, from the one that closed the pass on
        uint64_t controls = 0;  // outside the tile
        size_t ahead = 0;       // blocks looked at behind the one that closed the pass
        for (size_t i = first; i < nb && sel.gates.size() < kMaxBlocksPerPass; ++i) {
            if (held != 0 && ((moves_from[i] & ~held) == 0 || ++ahead > kMaxAhead)) break;
            if (done[i]) continue;
            const uint64_t mask = blocks[i].mask();
            uint64_t s2 = smask, d2 = dmask;
            // A CX needs its target in the tile; its control may be read outside it.
            const int kind = kinds[i];
            const bool cx = kind == TK_SW13 || kind == TK_SW23;
            const uint64_t control = cx ? uint64_t{1} << blocks[i].q[kind == TK_SW13 ? 0 : 1] : 0;
            if (diagonal_any_operand(blocks[i], is_param(i))) d2 |= mask;
            else if (cx && (s2 & control) == 0 && std::popcount(controls | control) <= static_cast<int>(cop::kMaxMapControls)) {
                s2 |= mask & ~control;
                d2 |= control;
            } else s2 |= mask;
            const bool fits = static_cast<uint32_t>(std::popcount(s2)) <= mt &&
                              outside(s2, d2) <= static_cast<int>(kMaxGlobalQubits) &&
                              (staged + staged_of(blocks[i], kind >= 0) <= kMaxStagedBytes || sel.gates.empty());
            if (!fits || (held != 0 && (!moves[i] || (mask & held) != 0))) {
                // (A move that does not fit closes the pass as any block does,
                // and no other move passes it.)
                if (held == 0 && moves[i]) break;
                held |= mask;
                continue;
            }
            staged += staged_of(blocks[i], kind >= 0);
            smask = s2;
            dmask = d2;
            if (cx && (s2 & control) == 0) controls |= control;
            sel.gates.push_back(static_cast<uint32_t>(i));
            done[i] = 1;
        }
        while (first < nb && done[first]) ++first;
        // Pad the tile to exactly mt qubits: first with the diagonals'
        // operands the global limit leaves out, then with the lowest unused
        // qubits (longer contiguous runs per tile).
        for (uint64_t rest = dmask & ~smask; std::popcount(rest) > static_cast<int>(kMaxGlobalQubits);
             rest &= rest - 1)
            smask |= rest & (~rest + 1);
        for (uint32_t q = 0; q < n && static_cast<uint32_t>(std::popcount(smask)) < mt; ++q)
            smask |= uint64_t{1} << q;
        sel.smask = smask;
        sel.gmask = dmask & ~smask;
        passes.push_back(std::move(sel));
    }
    return passes;
}

uint32_t push_matrix(std::vector<double>& data, const std::vector<Cd>& m) {
    const uint32_t off = static_cast<uint32_t>(data.size());
    for (const Cd& c : m) {
        data.push_back(c.real());
        data.push_back(c.imag());
    }
    return off;
}

}  // namespace

// Thread-bit order for a phase whose register bits are `reg` (tile-local
// positions): the first three thread bits get distinct residues mod 3 when
// possible, so that the eight threads of a quarter warp hit eight distinct
// 16-byte bank groups under the kernel's XOR-fold swizzle.
void thread_bit_order(uint32_t m, const uint32_t* reg, uint32_t nreg, uint8_t* tperm, uint8_t& nthread,
                      const TileMap* map, bool slots8) {
    std::vector<uint32_t> free_pos;
    for (uint32_t p = 0; p < m; ++p)
        if (std::find(reg, reg + nreg, p) == reg + nreg) free_pos.push_back(p);
    std::vector<uint32_t> order;
    const bool by_place = map != nullptr && !map->identity();
    if (by_place) {
        // The bank groups of a slot are its low bits (16-byte slots: three,
        // 8-byte: four), linear in the place: bits whose places have
        // independent ones first, by elimination.
        const uint32_t want = slots8 ? 4 : 3, low = (1u << want) - 1;
        uint32_t basis[4] = {0, 0, 0, 0};
        for (uint32_t p : free_pos) {
            if (order.size() == want) break;
            uint32_t v = (slots8 ? swz8(map->col[p]) : swz(map->col[p])) & low;
            for (uint32_t b = want; b-- > 0;) {
                if (!((v >> b) & 1u)) continue;
                if (basis[b] == 0) {
                    basis[b] = v;
                    order.push_back(p);
                    break;
                }
                v ^= basis[b];
            }
        }
    } else for (uint32_t res = 0; res < 3; ++res) {
        for (uint32_t p : free_pos)
            if (p % 3 == res && std::find(order.begin(), order.end(), p) == order.end()) {
                order.push_back(p);
                break;
            }
    }
    if (order.size() < 3 && !by_place) order.clear();
    for (uint32_t p : free_pos)
        if (std::find(order.begin(), order.end(), p) == order.end()) order.push_back(p);
    nthread = static_cast<uint8_t>(order.size());
    for (size_t i = 0; i < order.size(); ++i) tperm[i] = static_cast<uint8_t>(order[i]);
}

// Passes over a topological order of the blocks' dependencies (two blocks
// depend when they share a qubit; blocks on disjoint qubits commute), for
// the paths that are not bitwise the reference's sweep (complex64).  Each
// pass picks its tile greedily: the qubits of the earliest unapplied block,
// the fixed low qubits, then one qubit at a time the one that lets the most
// blocks run (ties: the one most blocked blocks wait for).  Inside the pass
// the blocks are ordered phase by phase: every ready block that a register
// set of four qubits (or no register at all: diagonals) can take, then the
// next set from the ready dense blocks, so the kernel changes phase rarely.
// Exact permutations need no registers either, but end the phase they come
// in (the amplitudes' places change), so they wait until no other block of
// the pass is ready.  Not in a pass that is rewritten for the tensor cores
// (tc_blocks: which blocks can be, in a program for them): there they are part
// of a phase's matrix like any other block, and waiting would spread them over
// more phases (81 layouts instead of 75 for a 26-qubit RY/RZ + CX ansatz,
// unfused).
std::vector<PassSel> select_passes_commuting(const std::vector<Block>& blocks, uint32_t n, uint32_t m,
                                             uint32_t fixed_low, const std::vector<int8_t>& kinds,
                                             const std::vector<uint8_t>* tc_blocks) {
    std::vector<PassSel> passes;
    uint32_t widest = 1;
    for (const Block& b : blocks) widest = std::max(widest, b.k);
    const uint32_t mt = std::min(m, n);
    if (widest > mt) throw std::invalid_argument("a block is wider than the tile");
    const uint32_t fixed = std::min(fixed_low, mt - widest);
    const uint32_t nb = static_cast<uint32_t>(blocks.size());
    std::vector<std::vector<uint32_t>> lists(n);
    std::vector<uint8_t> moves(nb, 0), none(nb, 0);
    bool mapped = false;
    for (uint32_t i = 0; i < nb; ++i) {
        moves[i] = kinds[i] >= 0;
        mapped = mapped || moves[i];
    }
    const bool tc = tc_blocks != nullptr && std::find(tc_blocks->begin(), tc_blocks->end(), 0) == tc_blocks->end();
    const Staged staged_of{mt, mapped, true, tc};
    std::vector<size_t> stages(nb);  // (looked at for every candidate below)
    for (uint32_t i = 0; i < nb; ++i) stages[i] = staged_of(blocks[i], moves[i] && tc_blocks == nullptr);
    for (uint32_t i = 0; i < nb; ++i)
        for (uint32_t t = 0; t < blocks[i].k; ++t) lists[blocks[i].q[t]].push_back(i);
    std::vector<uint32_t> head(n, 0);
    auto at_head = [&](const std::vector<uint32_t>& h, uint32_t i) {
        for (uint32_t t = 0; t < blocks[i].k; ++t) {
            const uint32_t y = blocks[i].q[t];
            if (h[y] >= lists[y].size() || lists[y][h[y]] != i) return false;
        }
        return true;
    };
    // Blocks that can run inside tile s from heads h, in a dependency order
    // (h advances past them); stops at the pass limits when `limit`.  Only
    // the heads of the qubits in `from` are looked at first: where h is already
    // past everything that runs in s without qubit x, x alone is enough, which
    // is how a candidate is tried below (a whole closure for each was most of
    // the time a plan took).
    std::vector<uint32_t> work;
    auto closure = [&](uint64_t s, std::vector<uint32_t>& h, std::vector<uint32_t>* out, bool limit, uint64_t from) {
        uint32_t count = 0;
        size_t staged = staged_of.base();
        work.clear();
        for (uint32_t x = 0; x < n; ++x)
            if ((from >> x) & 1u) work.push_back(x);
        while (!work.empty()) {
            const uint32_t x = work.back();
            work.pop_back();
            if (h[x] >= lists[x].size()) continue;
            const uint32_t i = lists[x][h[x]];
            if ((blocks[i].mask() & ~s) != 0 || !at_head(h, i)) continue;
            if (limit && (count >= kMaxBlocksPerPass ||
                          (count > 0 && staged + stages[i] > kMaxStagedBytes)))
                break;
            staged += stages[i];
            ++count;
            if (out) out->push_back(i);
            for (uint32_t t = 0; t < blocks[i].k; ++t) {
                ++h[blocks[i].q[t]];
                work.push_back(blocks[i].q[t]);
            }
        }
        return count;
    };
    uint32_t applied = 0, first = 0;
    std::vector<uint8_t> done(nb, 0);
    std::vector<uint32_t> h, base;
    while (applied < nb) {
        while (done[first]) ++first;
        uint64_t s = blocks[first].mask();
        for (uint32_t q = 0; q < fixed; ++q) s |= uint64_t{1} << q;
        base = head;
        uint64_t base_runs = closure(s, base, nullptr, false, s);
        while (static_cast<uint32_t>(std::popcount(s)) < mt) {
            uint64_t best_score = 0;
            uint32_t best = n;
            for (uint32_t x = 0; x < n; ++x) {
                if ((s >> x) & 1u) continue;
                h = base;
                const uint64_t runs = base_runs + closure(s | (uint64_t{1} << x), h, nullptr, false, uint64_t{1} << x);
                // Blocked blocks at the tile's heads that wait for x.
                uint32_t waits = 0;
                for (uint32_t y = 0; y < n; ++y)
                    if (((s >> y) & 1u) && head[y] < lists[y].size() &&
                        ((blocks[lists[y][head[y]]].mask() >> x) & 1u))
                        ++waits;
                const uint64_t score = (runs << 16) | waits;
                if (best == n || score > best_score) {
                    best_score = score;
                    best = x;
                }
            }
            s |= uint64_t{1} << best;
            base_runs += closure(s, base, nullptr, false, uint64_t{1} << best);
        }
        std::vector<uint32_t> members;
        h = head;
        closure(s, h, &members, true, s);
        if (members.empty()) throw std::logic_error("tile selection made no progress");
        // Phase-by-phase order of the members.
        PassSel sel;
        sel.smask = s;
        std::vector<uint8_t> in_pass(nb, 0);
        bool simt = tc_blocks == nullptr;
        for (uint32_t i : members) {
            in_pass[i] = 1;
            simt = simt || !(*tc_blocks)[i];
        }
        const std::vector<uint8_t>& waits = simt ? moves : none;
        std::vector<uint32_t> ph = head, sim, grown;
        std::vector<uint8_t> sim_in, grown_in;
        // Runs every member that register set `regs` can take (diagonals and
        // wide blocks need none), from heads hh, in waves: the ready dense
        // blocks, then the ready diagonals (so that the diagonals of one
        // layer are consecutive and merge), and so on; returns the dense
        // ones run.
        auto run = [&](uint64_t regs, std::vector<uint32_t>& hh, std::vector<uint8_t>& in, std::vector<uint32_t>* out) {
            uint32_t dense = 0;
            for (bool any = true; any;) {
                any = false;
                for (const bool diag : {false, true}) {
                    work.clear();
                    for (uint32_t x = 0; x < n; ++x)
                        if ((s >> x) & 1u) work.push_back(x);
                    while (!work.empty()) {
                        const uint32_t x = work.back();
                        work.pop_back();
                        if (hh[x] >= lists[x].size()) continue;
                        const uint32_t i = lists[x][hh[x]];
                        const Block& b = blocks[i];
                        if (!in[i] || b.diagonal != diag || waits[i] || !at_head(hh, i) ||
                            !(b.diagonal || b.k > 2 || (b.mask() & ~regs) == 0))
                            continue;
                        in[i] = 0;
                        any = true;
                        if (!b.diagonal && b.k <= 2) ++dense;
                        if (out) out->push_back(i);
                        for (uint32_t t = 0; t < b.k; ++t) {
                            ++hh[b.q[t]];
                            work.push_back(b.q[t]);
                        }
                    }
                }
            }
            return dense;
        };
        // The dense blocks that `regs` lets run from heads hh (which advance, as
        // `in` does), starting at qubit x: the same set as run's, in any order.
        auto count_from = [&](uint64_t regs, uint32_t x, std::vector<uint32_t>& hh, std::vector<uint8_t>& in) {
            uint32_t dense = 0;
            work.assign(1, x);
            while (!work.empty()) {
                const uint32_t y = work.back();
                work.pop_back();
                if (hh[y] >= lists[y].size()) continue;
                const uint32_t i = lists[y][hh[y]];
                const Block& b = blocks[i];
                if (!in[i] || waits[i] || !at_head(hh, i) || !(b.diagonal || b.k > 2 || (b.mask() & ~regs) == 0)) continue;
                in[i] = 0;
                if (!b.diagonal && b.k <= 2) ++dense;
                for (uint32_t t = 0; t < b.k; ++t) {
                    ++hh[b.q[t]];
                    work.push_back(b.q[t]);
                }
            }
            return dense;
        };
        size_t left = members.size();
        uint64_t regs = 0;
        for (;;) {
            const size_t before = sel.gates.size();
            run(regs, ph, in_pass, &sel.gates);
            left -= sel.gates.size() - before;
            if (left == 0) break;
            // Next register set: grown one qubit at a time by the qubit that
            // lets the most dense blocks run (ties: the one most ready dense
            // blocks use, then the lowest).
            uint64_t cand = 0;
            for (uint32_t i : members)
                if (in_pass[i] && !blocks[i].diagonal && blocks[i].k <= 2 && !waits[i]) cand |= blocks[i].mask();
            // Nothing but permutations ready: those that are.
            bool ready = false;
            for (uint32_t i : members)
                ready = ready || (in_pass[i] && !blocks[i].diagonal && blocks[i].k <= 2 && !waits[i] && at_head(ph, i));
            if (!ready) {
                bool any = false;
                for (bool again = true; again;) {
                    again = false;
                    for (uint32_t x = 0; x < n; ++x) {
                        if (!((s >> x) & 1u) || ph[x] >= lists[x].size()) continue;
                        const uint32_t i = lists[x][ph[x]];
                        if (!in_pass[i] || !waits[i] || !at_head(ph, i)) continue;
                        in_pass[i] = 0;
                        again = any = true;
                        sel.gates.push_back(i);
                        --left;
                        for (uint32_t t = 0; t < blocks[i].k; ++t) ++ph[blocks[i].q[t]];
                    }
                }
                if (any && left == 0) break;
                if (any) {
                    regs = 0;
                    continue;
                }
            }
            regs = 0;
            grown = ph;  // the heads after what the registers chosen so far let run
            grown_in = in_pass;
            uint64_t grown_runs = 0;
            for (uint32_t r = 0; r < kRegQubits && (cand & ~regs) != 0; ++r) {
                uint64_t best_score = 0;
                uint32_t best = n;
                for (uint32_t x = 0; x < n; ++x) {
                    if (!((cand >> x) & 1u) || ((regs >> x) & 1u)) continue;
                    sim = grown;
                    sim_in = grown_in;
                    const uint64_t runs = grown_runs + count_from(regs | (uint64_t{1} << x), x, sim, sim_in);
                    uint32_t uses = 0;
                    for (uint32_t i : members)
                        if (in_pass[i] && !blocks[i].diagonal && blocks[i].k <= 2 && !waits[i] &&
                            ((blocks[i].mask() >> x) & 1u) && at_head(ph, i))
                            ++uses;
                    const uint64_t score = (runs << 16) | uses;
                    if (best == n || score > best_score) {
                        best_score = score;
                        best = x;
                    }
                }
                regs |= uint64_t{1} << best;
                grown_runs += count_from(regs, best, grown, grown_in);
            }
            if (regs == 0) throw std::logic_error("phase ordering made no progress");
        }
        for (uint32_t i : sel.gates) done[i] = 1;
        applied += static_cast<uint32_t>(sel.gates.size());
        head = ph;
        passes.push_back(std::move(sel));
    }
    return passes;
}

TileProgram plan_tile_program(const std::vector<Block>& all, uint32_t n, uint32_t m, uint32_t fixed_low,
                              const std::vector<uint8_t>* all_parametric, bool commuting, bool split, bool latency) {
    // The blocks as they are planned: origin[i] the caller's block that part i
    // belongs to, last[i] whether it completes it.
    std::vector<Block> parts;
    std::vector<uint8_t> part_flags, last;
    std::vector<uint32_t> origin;
    for (size_t i = 0; i < all.size() && split && !latency; ++i) {
        if (origin.empty() && (all[i].k != 2 || all[i].diagonal)) continue;
        Block first, second;
        const uint8_t flags = all_parametric ? (*all_parametric)[i] : uint8_t{0};
        const bool two = !(flags & kParamBlock) && move_kind(all[i]) < 0 && split_block(all[i], first, second);
        if (two && parts.empty()) {  // from here on the parts are a list of their own
            parts.assign(all.begin(), all.begin() + static_cast<long>(i));
            for (uint32_t j = 0; j < i; ++j) {
                origin.push_back(j);
                last.push_back(1);
                part_flags.push_back(all_parametric ? (*all_parametric)[j] : uint8_t{0});
            }
            if (i == 0) parts.reserve(all.size() + 1);
        }
        if (two) {
            for (Block* p : {&first, &second}) {
                if (p->diagonal && p->k == 2) continue;  // the identity
                parts.push_back(std::move(*p));
                origin.push_back(static_cast<uint32_t>(i));
                last.push_back(0);
                part_flags.push_back(0);
            }
            last.back() = 1;
        } else if (!origin.empty()) {
            parts.push_back(all[i]);
            origin.push_back(static_cast<uint32_t>(i));
            last.push_back(1);
            part_flags.push_back(flags);
        }
    }
    const bool whole = origin.empty();
    const std::vector<Block>& blocks = whole ? all : parts;
    const std::vector<uint8_t>* parametric = whole || all_parametric == nullptr ? all_parametric : &part_flags;
    auto origin_of = [&](uint32_t i) { return whole ? i : origin[i]; };
    if (m < kMinTileQubits || m > kMaxTileQubitsC64) throw std::invalid_argument("tile width out of range");
    TileProgram prog;
    const uint32_t mt = std::min(m, n);
    if (mt < kRegQubits) throw std::invalid_argument("state too small for the tile kernel");
    if (commuting && !split)
        for (const Block& b : all) prog.tc_blocks.push_back(tc_convertible(b));
    std::vector<int8_t> kinds(blocks.size());  // move_kind; parametric blocks have none
    for (size_t i = 0; i < blocks.size(); ++i)
        kinds[i] = parametric != nullptr && ((*parametric)[i] & kParamBlock) != 0
                       ? int8_t{-1}
                       : static_cast<int8_t>(move_kind(blocks[i]));
    const std::vector<PassSel> sels =
        commuting ? select_passes_commuting(blocks, n, mt, fixed_low, kinds, split ? nullptr : &prog.tc_blocks)
                  : select_passes(blocks, n, mt, fixed_low, parametric, kinds);
    prog.c64 = commuting;
    prog.param_offsets.assign(all.size(), 0);
    auto param_flags = [&](uint32_t bi) -> uint8_t { return parametric ? (*parametric)[bi] : uint8_t{0}; };
    // A parametric block's data goes to the per-binding record.
    auto push_param = [&](uint32_t bi, uint32_t doubles) {
        const uint32_t off = prog.param_stride;
        prog.param_offsets[origin_of(bi)] = off;
        prog.param_stride += (doubles + 1) & ~1u;  // keep 16-byte alignment
        return off;
    };
    // The caller's blocks in an order of whole blocks that the parts' order
    // amounts to: one is listed when it is complete and every earlier block on
    // its qubits is.  Returns how many that made.  (Where no block is in parts,
    // the order they are planned in is that order.)
    std::vector<std::vector<uint32_t>> waiting(whole ? 0 : n);  // per qubit, latest block first
    for (uint32_t i = whole ? 0 : static_cast<uint32_t>(all.size()); i-- > 0;)
        for (uint32_t t = 0; t < all[i].k; ++t) waiting[all[i].q[t]].push_back(i);
    std::vector<uint8_t> ready(whole ? 0 : all.size(), 0);
    std::vector<uint32_t> look;
    auto complete = [&](uint32_t i) {
        uint32_t listed = 0;
        if (whole) {
            prog.order.push_back(i);
            prog.order_pass.push_back(static_cast<uint32_t>(prog.passes.size()));
            return uint32_t{1};
        }
        ready[i] = 1;
        look.assign(1, i);
        while (!look.empty()) {
            const uint32_t b = look.back();
            look.pop_back();
            bool first = ready[b] != 0;
            for (uint32_t t = 0; t < all[b].k && first; ++t)
                first = !waiting[all[b].q[t]].empty() && waiting[all[b].q[t]].back() == b;
            if (!first) continue;
            prog.order.push_back(b);
            prog.order_pass.push_back(static_cast<uint32_t>(prog.passes.size()));
            ++listed;
            for (uint32_t t = 0; t < all[b].k; ++t) waiting[all[b].q[t]].pop_back();
            for (uint32_t t = 0; t < all[b].k; ++t)
                if (!waiting[all[b].q[t]].empty()) look.push_back(waiting[all[b].q[t]].back());
        }
        return listed;
    };
    for (const PassSel& sel : sels) {
        TilePass pass;
        pass.m = mt;
        pass.smask = sel.smask;
        pass.gmask = sel.gmask;
        pass.prog_begin = static_cast<uint32_t>(prog.instrs.size());
        pass.sdata_begin = static_cast<uint32_t>(prog.data.size());
        auto push_staged = [&](const std::vector<Cd>& m) {
            return push_matrix(prog.data, m) - pass.sdata_begin;
        };

        bool open = false;
        TileMap map;
        uint32_t reg[kRegQubits];
        for (uint32_t r = 0; r < kRegQubits; ++r) reg[r] = r;
        auto in_reg = [&](uint32_t p) -> int {
            for (uint32_t s = 0; s < kRegQubits; ++s)
                if (reg[s] == p) return static_cast<int>(s);
            return -1;
        };
        auto close_phase = [&]() {
            if (open) {
                TileInstr e{};
                e.op = TOP_END;
                prog.instrs.push_back(e);
                open = false;
            }
        };
        // Opens a phase whose registers hold `first` (in order), filled from
        // the dense 1q/2q blocks that follow position `from` in this pass.
        auto open_phase = [&](const std::vector<uint32_t>& first, size_t from) {
            close_phase();
            std::vector<uint32_t> r(first);
            for (size_t j = from; j < sel.gates.size() && r.size() < kRegQubits; ++j) {
                const Block& b = blocks[sel.gates[j]];
                if (kinds[sel.gates[j]] >= 0) break;  // the phase ends there
                if (b.diagonal || b.k > 2) continue;
                bool fits = true;
                uint32_t extra = 0;
                for (uint32_t t = 0; t < b.k; ++t)
                    if (std::find(r.begin(), r.end(), local_pos(sel.smask, b.q[t])) == r.end()) ++extra;
                if (r.size() + extra > kRegQubits) fits = false;
                if (!fits) continue;
                for (uint32_t t = 0; t < b.k; ++t) {
                    const uint32_t p = local_pos(sel.smask, b.q[t]);
                    if (std::find(r.begin(), r.end(), p) == r.end()) r.push_back(p);
                }
            }
            for (uint32_t p = 0; p < mt && r.size() < kRegQubits; ++p)
                if (std::find(r.begin(), r.end(), p) == r.end()) r.push_back(p);
            for (uint32_t s = 0; s < kRegQubits; ++s) reg[s] = r[s];
            TileInstr ph{};
            ph.op = TOP_PHASE;
            for (uint32_t s = 0; s < kRegQubits; ++s) ph.pos[s] = static_cast<uint8_t>(reg[s]);
            thread_bit_order(mt, reg, kRegQubits, ph.tperm, ph.nthread, &map, commuting);
            prog.instrs.push_back(ph);
            open = true;
        };

        // A small diagonal's operand sources, decided here once: pos[4 + b]
        // = 0x80 | register slot, or the operand's tile bit (a thread bit).
        auto encode_sources = [&](TileInstr& g, uint32_t k) {
            for (uint32_t t = 0; t < k; ++t) {
                const int slot = in_reg(g.pos[t]);
                g.pos[4 + t] = static_cast<uint8_t>(slot >= 0 ? (0x80u | static_cast<uint32_t>(slot)) : g.pos[t]);
            }
        };
        for (size_t j = 0; j < sel.gates.size(); ++j) {
            const Block& b = blocks[sel.gates[j]];
            const uint32_t dim = 1u << b.k;
            if (whole || last[sel.gates[j]]) pass.gates += complete(origin_of(sel.gates[j]));
            TileInstr g{};
            g.k = static_cast<uint8_t>(b.k);
            const int move = kinds[sel.gates[j]];
            if (move >= 0) {
                close_phase();
                g.op = TOP_MOVE;
                g.kind = static_cast<uint8_t>(move);
                for (uint32_t t = 0; t < b.k; ++t)
                    g.pos[t] = static_cast<uint8_t>(operand_pos(sel.smask, sel.gmask, b.q[t]));
                map.move(g);
                prog.instrs.push_back(g);
                continue;
            }
            if (b.diagonal) {
                if (!open) open_phase({}, j + 1);
                g.op = TOP_DIAG;
                for (uint32_t t = 0; t < b.k; ++t)
                    g.pos[t] = static_cast<uint8_t>(operand_pos(sel.smask, sel.gmask, b.q[t]));
                std::vector<Cd> d(dim);
                for (uint32_t i = 0; i < dim; ++i) d[i] = b.m[i * dim + i];
                if (param_flags(sel.gates[j]) & kParamBlock) {
                    g.nthread = 1;
                    g.data = push_param(sel.gates[j], 2 * dim);
                    g.kind = b.k <= 2 ? TK_DSMALL : TK_GEN;
                    if (b.k <= 2) {
                        for (uint32_t i = 0; i < dim; ++i) g.aux |= 2u << (2 * i);  // every entry multiplies
                        encode_sources(g, b.k);
                    }
                    prog.fp64_per_amp += 6;
                    prog.instrs.push_back(g);
                    continue;
                }
                g.data = push_staged(d);
                if (b.k <= 2) {
                    // Entry classes: (1,0) copies, (-1,0) negates, the rest multiply.
                    g.kind = TK_DSMALL;
                    uint32_t gen = 0;
                    for (uint32_t i = 0; i < dim; ++i) {
                        uint32_t cls = 2;
                        if (d[i].imag() == 0.0 && d[i].real() == 1.0) cls = 0;
                        else if (d[i].imag() == 0.0 && d[i].real() == -1.0) cls = 1;
                        if (cls == 2) ++gen;
                        g.aux |= cls << (2 * i);
                    }
                    prog.fp64_per_amp += (6 * gen + dim - 1) / dim;
                    encode_sources(g, b.k);
                } else {
                    g.kind = TK_GEN;
                    prog.fp64_per_amp += 6;
                }
                prog.instrs.push_back(g);
                continue;
            }
            if (b.k <= 2) {
                int slot[2] = {-1, -1};
                bool have = open;
                for (uint32_t t = 0; t < b.k && have; ++t) {
                    slot[t] = in_reg(local_pos(sel.smask, b.q[t]));
                    if (slot[t] < 0) have = false;
                }
                if (!have) {
                    std::vector<uint32_t> first;
                    for (uint32_t t = 0; t < b.k; ++t) first.push_back(local_pos(sel.smask, b.q[t]));
                    open_phase(first, j + 1);
                    for (uint32_t t = 0; t < b.k; ++t) slot[t] = in_reg(local_pos(sel.smask, b.q[t]));
                }
                g.op = b.k == 1 ? TOP_G1 : TOP_G2;
                g.pos[0] = static_cast<uint8_t>(slot[0]);
                if (b.k == 2) g.pos[1] = static_cast<uint8_t>(slot[1]);
                // Specialisations, each exact up to the sign of zero results
                // (normalised at the store): monomial rows, real entries.
                const uint8_t pf = param_flags(sel.gates[j]);
                bool mono = (pf & kParamBlock) == 0;
                uint32_t aux = 0;
                for (uint32_t r = 0; r < dim && mono; ++r) {
                    const int s = mono_src(b.m, dim, r);
                    if (s == -2) {
                        mono = false;
                        break;
                    }
                    aux |= static_cast<uint32_t>(s < 0 ? 7 : s) << (3 * r);
                }
                if (mono) {
                    g.kind = TK_MONO;
                    g.aux = aux;
                    prog.fp64_per_amp += 6;
                } else if (b.k == 1) {
                    bool all_real = is_real(b.m[0]) && is_real(b.m[1]) && is_real(b.m[2]) && is_real(b.m[3]);
                    bool m00_real = is_real(b.m[0]);
                    if (pf & kParamBlock) {  // what holds for every binding
                        all_real = (pf & kParamAllReal) != 0;
                        m00_real = (pf & kParamM00Real) != 0;
                    }
                    if (all_real) {
                        g.kind = TK_REAL;
                        prog.fp64_per_amp += 6;
                    } else if (m00_real) {
                        g.kind = TK_U3;
                        prog.fp64_per_amp += 12;
                    } else {
                        g.kind = TK_GEN;
                        prog.fp64_per_amp += 14;
                    }
                } else if (!commuting && (pf & kParamBlock) == 0 && is_cross(b)) {
                    // 6 FP64 operations per amplitude instead of 30.  Slots in
                    // ascending order: swapped operands exchange indices 1 and 2.
                    g.kind = TK_CROSS;
                    const uint32_t one = g.pos[0] < g.pos[1] ? 1 : 2, two = 3 - one;
                    if (g.pos[0] > g.pos[1]) std::swap(g.pos[0], g.pos[1]);
                    auto e = [&](uint32_t r, uint32_t c) { return b.m[4 * r + c].real(); };
                    g.data = push_staged({Cd(e(0, 0), e(0, 3)), Cd(e(3, 0), e(3, 3)), Cd(e(one, one), e(one, two)),
                                          Cd(e(two, one), e(two, two))});
                    prog.fp64_per_amp += 6;
                    prog.instrs.push_back(g);
                    continue;
                } else {
                    g.kind = TK_GEN;
                    prog.fp64_per_amp += 30;
                }
                if (pf & kParamBlock) {
                    g.nthread = 1;
                    g.data = push_param(sel.gates[j], 2 * dim * dim);
                } else {
                    g.data = push_staged(b.m);
                }
                prog.instrs.push_back(g);
                continue;
            }
            // Wider dense block: from shared memory, as a phase of its own, with
            // the amplitudes at their own index.
            close_phase();
            if (!map.identity()) {
                open_phase({}, sel.gates.size());
                prog.instrs.back().kind = 1;  // settle
                close_phase();
                map = TileMap();
            }
            g.op = TOP_SMEM;
            pass.wide = true;
            for (uint32_t t = 0; t < b.k; ++t) g.pos[t] = static_cast<uint8_t>(local_pos(sel.smask, b.q[t]));
            if (param_flags(sel.gates[j]) & kParamBlock)
                throw std::invalid_argument("parametric blocks wider than 2 qubits are not batched");
            g.data = push_matrix(prog.gdata, b.m);
            prog.instrs.push_back(g);
            prog.fp64_per_amp += 8ull * dim - 2;
        }
        close_phase();
        pass.prog_count = static_cast<uint32_t>(prog.instrs.size()) - pass.prog_begin;
        pass.sdata_count = static_cast<uint32_t>(prog.data.size()) - pass.sdata_begin;
        prog.passes.push_back(pass);
    }
    encode_compact(prog);
    // Short passes all run the kernel with the map where one of them needs it:
    // going from one kernel to the other costs more than the 1 % that the map
    // costs the rest (kOneKernelQubits).
    if (n <= kOneKernelQubits) {
        bool any = false;
        for (const TilePass& p : prog.passes) any = any || p.mapped;
        for (TilePass& p : prog.passes) p.mapped = any;
    }
    for (size_t i = 1; i < prog.passes.size() && !commuting; ++i)
        prog.passes[i].behind = prog.passes[i].wide == prog.passes[i - 1].wide;
    return prog;
}

}  // namespace mb2
