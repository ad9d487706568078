/*
 * encoder.cpp - postfix bytecode -> accumulator-machine record.
 *
 * Stage 1 (parse) walks the byte stream with the per-token checks of the reference evaluator
 * and specializer (projects/secant/s_cpu.c:193-414, s_cubin_specialize.c:1203-1368), in their
 * order, expanding routine calls in place with their arguments bound once.  It builds an
 * expression DAG (a routine argument used several times becomes a shared node).
 * Stage 2 (label, as the nodes are made) notes for every node by what its value depends on: nothing (literals), the
 * coefficient bank, the row, or both.
 * Stage 3 (emit) linearises the DAG for a machine with one accumulator: a binary node whose
 * other operand is a leaf costs one instruction, a node with two computed operands spills the
 * first through a slot.  The deeper operand is evaluated first (Sethi-Ullman order), which only
 * changes the order pure sub-expressions are computed in, never how values are rounded or
 * associated.  For the population evaluator the instructions go to up to four runs (record.h):
 * bank-only sub-expressions to the bank part, row-only ones to the shared row prelude (no toggle
 * reaches them) or the row prelude, the rest to the main part.
 */
#include "encoder.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace sb {

void EncodedBatch::clear() {
    programs.clear(); insns.clear(); patches.clear(); affines.clear(); lits.clear();
    max_insn = 1; max_extra = 0; max_slots = 0; max_patch = 0; max_hoisted = 0; max_cst = 0; max_btmp = 0;
    uses_scratch = false;
}

namespace {

/* ---- tokens ---------------------------------------------------------------------------- */

enum TokenKind : uint8_t { TK_COLUMN, TK_BANK, TK_AFFINE, TK_LITERAL, TK_TOGGLE, TK_ARG, TK_CALL, TK_RETURN, TK_OPERATION };

struct Token {
    TokenKind kind;
    uint8_t ways;   /* toggles: 2 or 4 */
    uint8_t arity;  /* operations */
    uint8_t node;   /* operations: 1 unary, 2 binary, 3 fma */
    uint8_t op;     /* SB_UN_* or SB_BIN_* */
    size_t width;
};

/* operations: {opcode, arity, SB_* code} */
struct OperationRow { uint8_t opcode, arity, code; };
constexpr OperationRow kOperations[] = {
    {SECANT_AST_INSTRUCTION_TYPE_ADD_F32, 2, SB_BIN_ADD},   {SECANT_AST_INSTRUCTION_TYPE_SUB_F32, 2, SB_BIN_SUB},
    {SECANT_AST_INSTRUCTION_TYPE_MUL_F32, 2, SB_BIN_MUL},   {SECANT_AST_INSTRUCTION_TYPE_DIV_F32, 2, SB_BIN_DIV},
    {SECANT_AST_INSTRUCTION_TYPE_MIN_F32, 2, SB_BIN_MIN},   {SECANT_AST_INSTRUCTION_TYPE_MAX_F32, 2, SB_BIN_MAX},
    {SECANT_AST_INSTRUCTION_TYPE_FMA_F32, 3, 0},
    {SECANT_AST_INSTRUCTION_TYPE_NEG_F32, 1, SB_UN_NEG},    {SECANT_AST_INSTRUCTION_TYPE_SQRT_F32, 1, SB_UN_SQRT},
    {SECANT_AST_INSTRUCTION_TYPE_RCP_F32, 1, SB_UN_RCP},    {SECANT_AST_INSTRUCTION_TYPE_ABS_F32, 1, SB_UN_ABS},
    {SECANT_AST_INSTRUCTION_TYPE_SIN_F32, 1, SB_UN_SIN},    {SECANT_AST_INSTRUCTION_TYPE_COS_F32, 1, SB_UN_COS},
    {SECANT_AST_INSTRUCTION_TYPE_EX2_F32, 1, SB_UN_EX2},    {SECANT_AST_INSTRUCTION_TYPE_LG2_F32, 1, SB_UN_LG2},
    {SECANT_AST_INSTRUCTION_TYPE_RSQRT_F32, 1, SB_UN_RSQRT}, {SECANT_AST_INSTRUCTION_TYPE_TANH_F32, 1, SB_UN_TANH},
    {SECANT_AST_INSTRUCTION_TYPE_EXP_F32, 1, SB_UN_EXP},    {SECANT_AST_INSTRUCTION_TYPE_LOG_F32, 1, SB_UN_LOG},
};

/* The float32 opcodes the evaluators accept (projects/secant/s_ast_internal.h:103-117). */
bool evaluable_opcode(unsigned op) {
    switch (op) {
    case SECANT_AST_INSTRUCTION_TYPE_AFFINE_BANK_F32: case SECANT_AST_INSTRUCTION_TYPE_COLUMN_F32:
    case SECANT_AST_INSTRUCTION_TYPE_BANK_CONSTANT_F32: case SECANT_AST_INSTRUCTION_TYPE_TOGGLE2_F32:
    case SECANT_AST_INSTRUCTION_TYPE_TOGGLE4_F32: case SECANT_AST_INSTRUCTION_TYPE_EXP_F32:
    case SECANT_AST_INSTRUCTION_TYPE_LOG_F32:
        return true;
    default:
        return op >= SECANT_AST_INSTRUCTION_TYPE_CONSTANT_BITS_F32 && op <= SECANT_AST_INSTRUCTION_TYPE_TANH_F32;
    }
}

/* What the first byte of a token says, by opcode: every program is walked twice (preflight, parser)
 * before its call can start, so the per-token work is one table row.  `status` comes before every
 * other check; a row that is an operation with arity 0 (NONE) decodes but cannot be evaluated. */
struct OpcodeTable {
    struct Row { Token token; SecantResult status; } row[256];
    OpcodeTable() {
        for (unsigned op = 0; op < 256; ++op) {
            const SecantAstInstruction first = (SecantAstInstruction)op;
            Token t{TK_OPERATION, 0, 0, 0, 0, secant_ast_instruction_size_get(&first)};
            SecantResult status = SECANT_SUCCESS;
            if (!t.width) status = SECANT_ERROR_BAD_PROGRAM;
            else if (!evaluable_opcode(op)) status = SECANT_ERROR_UNSUPPORTED_OP;
            switch (op) {
            case SECANT_AST_INSTRUCTION_TYPE_COLUMN_F32: t.kind = TK_COLUMN; break;
            case SECANT_AST_INSTRUCTION_TYPE_BANK_CONSTANT_F32: t.kind = TK_BANK; break;
            case SECANT_AST_INSTRUCTION_TYPE_AFFINE_BANK_F32: t.kind = TK_AFFINE; break;
            case SECANT_AST_INSTRUCTION_TYPE_CONSTANT_BITS_F32: t.kind = TK_LITERAL; break;
            case SECANT_AST_INSTRUCTION_TYPE_TOGGLE2_F32: t.kind = TK_TOGGLE; t.ways = 2; break;
            case SECANT_AST_INSTRUCTION_TYPE_TOGGLE4_F32: t.kind = TK_TOGGLE; t.ways = 4; break;
            case SECANT_AST_INSTRUCTION_TYPE_ROUTINE_ARG_F32: t.kind = TK_ARG; break;
            case SECANT_AST_INSTRUCTION_TYPE_ROUTINE_F32: t.kind = TK_CALL; break;
            case SECANT_AST_INSTRUCTION_TYPE_RETURN_F32: t.kind = TK_RETURN; break;
            default:
                for (const OperationRow& o : kOperations)
                    if (o.opcode == op) { t.arity = t.node = o.arity; t.op = o.code; }
            }
            row[op] = Row{t, status};
        }
    }
};
const OpcodeTable kTable;

/* Decodes one token and applies every check that needs no evaluation state: byte width, opcode
 * class, leaf index ranges, toggle bit ranges, finite affine payloads.  Both the runner's
 * preflight (projects/secant/s_cubin_runner.c:138-181) and the parser below start from it, so
 * the two cannot disagree on what a well-formed token is. */
inline SecantResult read_token(const SecantAstInstruction* ins, const ProgramRules& rules, Token* t) {
    const OpcodeTable::Row& row = kTable.row[ins[0]];
    *t = row.token;
    if (row.status != SECANT_SUCCESS) return row.status;
    bool good = true;
    switch (row.token.kind) {
    case TK_COLUMN: good = ins[1] < rules.num_columns; break;
    case TK_BANK: good = rules.banks_allowed && ins[1] < rules.num_constants; break;
    case TK_AFFINE:
        good = rules.banks_allowed && ins[1] < rules.num_constants && std::isfinite(secant_ast_affine_bank_scale_get(ins)) &&
               std::isfinite(secant_ast_affine_bank_offset_get(ins));
        break;
    case TK_TOGGLE:
        good = rules.banks_allowed && ins[1] < rules.toggle_bits &&
               (row.token.ways == 2 || (ins[2] < rules.toggle_bits && ins[2] != ins[1]));
        break;
    default: break;
    }
    return good ? SECANT_SUCCESS : SECANT_ERROR_BAD_PROGRAM;
}

inline bool direct_leaf(TokenKind k) { return k == TK_COLUMN || k == TK_BANK || k == TK_AFFINE || k == TK_LITERAL; }

/* ---- expression DAG -------------------------------------------------------------------- */

enum NodeType : uint8_t { N_COL, N_BANK, N_AFFINE, N_LIT, N_TOGGLE, N_UN, N_BIN, N_FMA };
/* What a value depends on, as bits: joining two classes is an or. */
enum ValueClass : uint8_t { VC_LITERAL = 0, VC_BANK = 1, VC_ROW = 2, VC_MIXED = 3 };

inline ValueClass join(ValueClass a, ValueClass b) { return (ValueClass)(a | b); }

struct Node {
    NodeType type = N_LIT;
    uint8_t op = 0;       /* SB_UN_* for N_UN, SB_BIN_{ADD,SUB,MUL,DIV,MIN,MAX} for N_BIN */
    uint8_t ways = 0;     /* toggle: 2 or 4 */
    uint8_t bit0 = 0, bit1 = 0xff;
    ValueClass cls = VC_LITERAL;
    bool toggled = false; /* a toggle lies somewhere below (or here): the value changes with the permutation */
    uint8_t seen = 0;     /* marks of collect() */
    int32_t child[4] = {-1, -1, -1, -1};
    uint32_t index = 0;   /* column / bank slot / affine entry */
    uint32_t bits = 0;    /* literal */
    int32_t uses = 0;     /* parents inside the run being emitted */
    int32_t pending = 0;  /* uses not yet emitted */
    int32_t slot = -1;    /* spill slot holding the value, once computed */
    int32_t su = 0;       /* slots needed to compute the node into the accumulator */
    int32_t hoisted = -1; /* per-row value the prelude left */
    int32_t entry = -1;   /* constant-table entry the bank part left */
    int32_t weight = 0;   /* rough instruction cost of the sub-expression */
};

unsigned arity_of(const Node& n) { return n.type > N_TOGGLE ? (unsigned)n.type - N_TOGGLE : 0u; } /* N_UN, N_BIN, N_FMA follow it */

/* rough executed-instruction weights used for scheduling (SbProgram::cost) and for choosing
 * which row-only sub-expressions are worth a hoist slot */
constexpr int unary_weight(unsigned op) {
    return op == SB_UN_NEG || op == SB_UN_ABS ? 1 : op == SB_UN_SIN || op == SB_UN_COS ? 18 : op == SB_UN_EXP || op == SB_UN_EX2 ? 9 : op == SB_UN_LOG ? 14 : 12;
}
constexpr int binary_weight(unsigned op) { return (op == SB_BIN_DIV || op == SB_BIN_RDIV) ? 11 : 1; }

/* What the parser does with a token: one branch decides between the kinds of leaves and operations (programs are
 * random to the processor, and a branch it guesses wrongly costs as much as the rest of a token). */
enum Step : uint8_t { STEP_COLUMN, STEP_BANK, STEP_AFFINE, STEP_LITERAL, STEP_TOGGLE, STEP_ARG, STEP_CALL, STEP_RETURN, STEP_UNARY, STEP_BINARY, STEP_FMA, STEP_NONE };
struct StepTable {
    struct Row { Step step; uint8_t op, ways, width; uint8_t status; int8_t weight; } row[256];
    StepTable() {
        for (unsigned op = 0; op < 256; ++op) {
            const OpcodeTable::Row& r = kTable.row[op];
            const Token& t = r.token;
            const Step operation = t.arity == 1 ? STEP_UNARY : t.arity == 2 ? STEP_BINARY : t.arity == 3 ? STEP_FMA : STEP_NONE;
            static const Step steps[] = {STEP_COLUMN, STEP_BANK, STEP_AFFINE, STEP_LITERAL, STEP_TOGGLE, STEP_ARG, STEP_CALL, STEP_RETURN};
            row[op] = Row{t.kind == TK_OPERATION ? operation : steps[t.kind], t.op, t.ways, (uint8_t)t.width, (uint8_t)r.status,
                          (int8_t)(t.arity == 1 ? unary_weight(t.op) : t.arity == 2 ? binary_weight(t.op) : 4)};
        }
    }
};
const StepTable kSteps;

struct Parser {
    const SecantAstProgramList& routines;
    const uint8_t* arity;
    const ProgramRules& rules;
    std::vector<Node>& nodes;
    std::vector<SbAffine>& affines; /* of this program */
    unsigned n_ops = 0;
    unsigned of_class[4] = {0, 0, 0, 0}; /* operations by what their value depends on */

    int leaf(NodeType type, ValueClass cls, uint32_t index, uint32_t bits) {
        nodes.emplace_back();
        Node& n = nodes.back();
        n.type = type; n.cls = cls; n.index = index; n.bits = bits;
        return (int)nodes.size() - 1;
    }
    /* An operation over the top of a stack, labelled with what its value depends on and what it costs (a shared value
     * counts once per parent): children exist before their parents, so one look at them is enough. */
    template <unsigned ARITY>
    int operation(NodeType type, const StepTable::Row& row, const int* children) {
        nodes.emplace_back();
        Node& n = nodes.back();
        n.type = type;
        n.op = row.op;
        int64_t w = row.weight;
        unsigned cls = 0, toggled = 0;
        for (unsigned i = 0; i < ARITY; ++i) {
            const Node& c = nodes[(size_t)children[i]];
            n.child[i] = children[i];
            cls |= c.cls;
            toggled |= c.toggled ? 1u : 0u;
            w += c.weight;
        }
        n.cls = (ValueClass)cls;
        n.toggled = toggled != 0;
        n.weight = (int32_t)std::min<int64_t>(w, INT32_MAX);
        ++n_ops;
        ++of_class[cls];
        return (int)nodes.size() - 1;
    }

    int affine_entry(uint32_t slot, float scale, float offset) {
        for (size_t i = 0; i < affines.size(); ++i)
            if (affines[i].slot == slot && !std::memcmp(&affines[i].scale, &scale, 4) &&
                !std::memcmp(&affines[i].offset, &offset, 4))
                return (int)i;
        affines.push_back(SbAffine{slot, scale, offset});
        return (int)affines.size() - 1;
    }

    /* One frame of the evaluator: its own value stack, arguments bound to nodes of the caller. */
    SecantResult frame(const SecantAstInstruction* code, const int* args, size_t num_args, unsigned depth, int* result) {
        int stack[SECANT_AST_MAX_STACK_DEPTH];
        size_t top = 0, leaves_in_a_row = 0;
        if (!code) return SECANT_ERROR_BAD_PROGRAM;
        const SecantAstInstruction* ins = code;
        const ValueClass column_class = rules.columns_are_slots ? VC_MIXED : VC_ROW;
        for (size_t n = 0; n < SECANT_AST_MAX_PROGRAM_INSTRUCTIONS; ++n) { /* the checks of read_token() first, in its order */
            const StepTable::Row row = kSteps.row[ins[0]];
            if (row.status != SECANT_SUCCESS) return (SecantResult)row.status;
            size_t leaves = 0;
            switch (row.step) {
            case STEP_COLUMN:
                if (ins[1] >= rules.num_columns) return SECANT_ERROR_BAD_PROGRAM;
                if (top == SECANT_AST_MAX_STACK_DEPTH) return SECANT_ERROR_STACK_OVERFLOW;
                stack[top++] = leaf(N_COL, column_class, ins[1], 0);
                leaves = leaves_in_a_row + 1;
                break;
            case STEP_BANK:
                if (!rules.banks_allowed || ins[1] >= rules.num_constants) return SECANT_ERROR_BAD_PROGRAM;
                if (top == SECANT_AST_MAX_STACK_DEPTH) return SECANT_ERROR_STACK_OVERFLOW;
                stack[top++] = leaf(N_BANK, VC_BANK, ins[1], 0);
                leaves = leaves_in_a_row + 1;
                break;
            case STEP_AFFINE: {
                const float scale = secant_ast_affine_bank_scale_get(ins), offset = secant_ast_affine_bank_offset_get(ins);
                if (!rules.banks_allowed || ins[1] >= rules.num_constants || !std::isfinite(scale) || !std::isfinite(offset)) return SECANT_ERROR_BAD_PROGRAM;
                if (top == SECANT_AST_MAX_STACK_DEPTH) return SECANT_ERROR_STACK_OVERFLOW;
                stack[top++] = leaf(N_AFFINE, VC_BANK, (uint32_t)affine_entry(ins[1], scale, offset), 0);
                leaves = leaves_in_a_row + 1;
                break;
            }
            case STEP_LITERAL:
                if (top == SECANT_AST_MAX_STACK_DEPTH) return SECANT_ERROR_STACK_OVERFLOW;
                stack[top++] = leaf(N_LIT, VC_LITERAL, 0, secant_ast_constant_bits_get(ins));
                leaves = leaves_in_a_row + 1;
                break;
            case STEP_ARG:
                if (!args || ins[1] >= num_args) return SECANT_ERROR_ROUTINE_ARG_IDX_OUT_OF_BOUNDS;
                if (top == SECANT_AST_MAX_STACK_DEPTH) return SECANT_ERROR_STACK_OVERFLOW;
                stack[top++] = args[ins[1]];
                break;
            case STEP_TOGGLE: {
                if (!rules.banks_allowed || ins[1] >= rules.toggle_bits || (row.ways == 4 && (ins[2] >= rules.toggle_bits || ins[2] == ins[1])))
                    return SECANT_ERROR_BAD_PROGRAM;
                if (leaves_in_a_row < row.ways || top < row.ways) return SECANT_ERROR_BAD_PROGRAM;
                nodes.emplace_back();
                Node& nd = nodes.back();
                nd.type = N_TOGGLE;
                nd.toggled = true;
                nd.ways = row.ways; nd.bit0 = ins[1]; nd.bit1 = row.ways == 4 ? ins[2] : 0xff;
                top -= row.ways;
                for (size_t i = 0; i < row.ways; ++i) {
                    nd.child[i] = stack[top + i];
                    nd.cls = join(nd.cls, nodes[(size_t)stack[top + i]].cls);
                }
                stack[top++] = (int)nodes.size() - 1;
                break;
            }
            case STEP_CALL: {
                if (ins[1] >= routines.count || !routines.items[ins[1]]) return SECANT_ERROR_ROUTINE_IDX_OUT_OF_BOUNDS;
                if (depth >= kRoutineDepth) return SECANT_ERROR_ROUTINE_DEPTH_EXCEEDED;
                const size_t want = arity[ins[1]];
                if (top < want) return SECANT_ERROR_STACK_UNDERFLOW;
                int value = -1;
                const SecantResult r = frame(routines.items[ins[1]], stack + (top - want), want, depth + 1, &value);
                if (r != SECANT_SUCCESS) return r;
                top -= want;
                stack[top++] = value;
                break;
            }
            case STEP_RETURN:
                if (top != 1u) return SECANT_ERROR_BAD_PROGRAM;
                *result = stack[0];
                return SECANT_SUCCESS;
            case STEP_UNARY:
                if (top < 1) return SECANT_ERROR_STACK_UNDERFLOW;
                stack[top - 1] = operation<1>(N_UN, row, stack + top - 1);
                break;
            case STEP_BINARY:
                if (top < 2) return SECANT_ERROR_STACK_UNDERFLOW;
                --top;
                stack[top - 1] = operation<2>(N_BIN, row, stack + top - 1);
                break;
            case STEP_FMA:
                if (top < 3) return SECANT_ERROR_STACK_UNDERFLOW;
                top -= 2;
                stack[top - 1] = operation<3>(N_FMA, row, stack + top - 1);
                break;
            default: return SECANT_ERROR_BAD_PROGRAM;
            }
            leaves_in_a_row = leaves;
            ins += row.width;
        }
        return SECANT_ERROR_BAD_PROGRAM;
    }
};

struct Operand {
    unsigned kind;
    unsigned index;
};

/* The instruction runs of a record.  The row prelude comes in two runs: values no toggle can change,
 * which an item that covers several permutations computes once, and values a toggle reaches. */
enum Run { RUN_BANK = 0, RUN_SHARED = 1, RUN_ROW = 2, RUN_MAIN = 3, NUM_RUNS = 4 };

struct InsnWeights {
    uint8_t of[256];
    constexpr InsnWeights() : of() {
        for (unsigned cs = 0; cs < 256; ++cs)
            of[cs] = (uint8_t)(cs >= SB_CASE_BIN && cs < SB_CASE_UN ? 1 + binary_weight((cs - SB_CASE_BIN) / SB_NUM_KINDS)
                             : cs >= SB_CASE_UN && cs < SB_CASE_FMA ? 1 + unary_weight(cs - SB_CASE_UN) : cs == SB_CASE_FMA ? 12 : 2);
    }
};
constexpr InsnWeights kInsnWeights;
inline unsigned insn_weight(const SbInsn& ins) { return kInsnWeights.of[ins.w0 & 0xffu]; }

struct LeafEntry { NodeType type; uint32_t key; int entry; };

/* Working storage of one encode_program() call.  Every thread keeps one: a program needs a dozen
 * small arrays, and making them anew for each program cost as much as filling them (5.9 us per
 * program of the 32-token, 16-slot kind on a 2.7 GHz Xeon; 3.0 us with the arrays kept, the nodes
 * labelled as they are parsed and each phase resetting only the nodes it reached; 2.2 with one branch per token,
 * classes joined by an or, and leaves counted where they are read). */
struct Scratch {
    std::vector<Node> nodes;
    std::vector<SbAffine> affines; /* of this program */
    std::vector<SbInsn> code[NUM_RUNS];
    std::vector<SbPatch> sites[NUM_RUNS]; /* SbPatch::insn is relative to the run until the record is assembled */
    std::vector<uint8_t> slot_busy;
    std::vector<int> touched;             /* nodes the phase being emitted reaches */
    std::vector<LeafEntry> leaf_entries;
    std::vector<int> bank_roots, row_roots, shared_roots, chosen;
    std::vector<SbInsn> fused;
    std::vector<uint8_t> is_site;
    std::vector<uint32_t> moved;

    void begin() {
        if (nodes.capacity() > 8192) *this = Scratch(); /* an unusually large program's storage is not kept */
        nodes.clear(); affines.clear(); slot_busy.clear(); touched.clear(); leaf_entries.clear();
        bank_roots.clear(); row_roots.clear(); shared_roots.clear(); chosen.clear();
        for (auto& c : code) c.clear();
        for (auto& c : sites) c.clear();
    }
};

/* Bookkeeping rule of the emitter: gen(id) leaves the value of node `id` in the accumulator and
 * never consumes a use; the instruction that reads a value (as its accumulator input or as its
 * operand) consumes one use of it.  A computed node with several parents is parked in a slot
 * right after it is computed; a slot is released when the last use of its node is consumed. */
struct Emitter {
    Scratch& mem;
    std::vector<Node>& nodes;
    const ProgramRules& rules;
    EncodedBatch& out;
    size_t lit_base;
    unsigned n_affine;
    std::vector<SbInsn> (&code)[NUM_RUNS];
    std::vector<SbPatch> (&sites)[NUM_RUNS];
    Run run = RUN_MAIN;
    std::vector<uint8_t>& slot_busy;
    unsigned slots_high = 0, btmp_high = 0;
    unsigned n_entries = 0, n_hoisted = 0;
    bool uses_scratch = false;
    SecantResult error = SECANT_SUCCESS;
    std::vector<LeafEntry>& leaf_entries;

    Emitter(Scratch& mem_, const ProgramRules& rules_, EncodedBatch& out_)
        : mem(mem_), nodes(mem_.nodes), rules(rules_), out(out_), lit_base(out_.lits.size()), n_affine((unsigned)mem_.affines.size()),
          code(mem_.code), sites(mem_.sites), slot_busy(mem_.slot_busy), leaf_entries(mem_.leaf_entries) {}

    static bool leaf_type(const Node& n) { return n.type <= N_TOGGLE; }
    /* a value that can be named as an operand without computing anything */
    bool ready(int id) const { return ready(nodes[id]); }
    bool ready(const Node& n) const {
        return leaf_type(n) || n.slot >= 0 || (run != RUN_BANK && n.hoisted >= 0) || n.entry >= 0;
    }

    /* Sub-expressions to move out of the main part: maximal computed nodes whose value depends on
     * the bank only (or on nothing), and maximal computed nodes that depend on the row only.
     * Inside a row-only expression, literal-only computed nodes still go to the bank part. */
    void collect(int id, bool inside_row, std::vector<int>& bank_roots, std::vector<int>& row_roots) {
        Node& n = nodes[id];
        const unsigned mark = inside_row ? 2u : 1u;
        if (leaf_type(n) || (n.seen & mark)) return;
        n.seen |= (uint8_t)mark;
        if (n.cls <= VC_BANK && rules.hoist_bank) {
            if (std::find(bank_roots.begin(), bank_roots.end(), id) == bank_roots.end()) bank_roots.push_back(id);
            return;
        }
        if (n.cls == VC_ROW && rules.hoist_row && !inside_row) {
            if (std::find(row_roots.begin(), row_roots.end(), id) == row_roots.end()) row_roots.push_back(id);
            inside_row = true;
        }
        const unsigned arity = arity_of(n);
        for (unsigned i = 0; i < arity; ++i) collect(n.child[i], inside_row, bank_roots, row_roots);
    }

    /* maximal computed row-only nodes below `id` that no toggle reaches */
    void collect_shared(int id, std::vector<int>& shared) {
        const Node& n = nodes[id];
        if (leaf_type(n)) return;
        if (n.cls == VC_ROW && !n.toggled) {
            if (std::find(shared.begin(), shared.end(), id) == shared.end()) shared.push_back(id);
            return;
        }
        const unsigned arity = arity_of(n);
        for (unsigned i = 0; i < arity; ++i) collect_shared(n.child[i], shared);
    }

    int alloc_slot() {
        for (size_t i = 0; i < slot_busy.size(); ++i)
            if (!slot_busy[i]) { slot_busy[i] = 1; return (int)i; }
        if (slot_busy.size() >= kMaxSlots) { error = SECANT_ERROR_REGISTER_OVERFLOW; return 0; }
        slot_busy.push_back(1);
        unsigned& high = run == RUN_BANK ? btmp_high : slots_high;
        if (slot_busy.size() > high) high = (unsigned)slot_busy.size();
        return (int)slot_busy.size() - 1;
    }

    /* Every hoisted expression and the main part are emitted as separate phases that share nothing
     * but hoisted values and table entries: parent counts, pending uses and slots start afresh, so
     * a node needed by two phases is simply computed in both (a slot written during one row pass
     * of the prelude could not be trusted by the main part of every bank group). */
    void begin_phase(Run r, int phase_root) {
        run = r;
        for (int id : mem.touched) { Node& n = nodes[id]; n.uses = 0; n.pending = 0; n.slot = -1; } /* of the phase before */
        mem.touched.clear();
        slot_busy.clear();
        if (r != RUN_BANK) slot_busy.assign(rules.reserved_slots, 1);
        prepare(phase_root);
        for (int id : mem.touched) nodes[id].pending = nodes[id].uses;
    }

    /* Counts parent references of every reachable node and computes how many slots each needs
     * while it is being evaluated (Sethi-Ullman numbers, DAG-agnostic estimate). */
    void prepare(int id) {
        Node& n = nodes[id]; /* (no node is made here) */
        if (n.uses++ > 0) return;
        mem.touched.push_back(id);
        if (ready(n)) { n.su = 0; return; }
        const auto need = [&](int child) { /* slots, or -1 where nothing has to be computed */
            Node& c = nodes[child];
            if (leaf_type(c)) {
                if (c.uses++ == 0) mem.touched.push_back(child);
                return -1;
            }
            prepare(child);
            return ready(c) ? -1 : c.su;
        };
        if (n.type == N_UN) {
            n.su = std::max(0, need(n.child[0]));
        } else if (n.type == N_BIN) {
            const int l = need(n.child[0]), r = need(n.child[1]);
            n.su = std::max(0, std::max(std::max(l, r), std::min(l, r) < 0 ? -1 : std::min(l, r) + 1));
        } else { /* the k-th operand evaluated, hungriest first, coexists with k parked predecessors */
            int of[3] = {need(n.child[0]), need(n.child[1]), need(n.child[2])};
            std::sort(of, of + 3, [](int a, int b) { return a > b; });
            n.su = 0;
            for (int i = 0; i < 3 && of[i] >= 0; ++i) n.su = std::max(n.su, of[i] + i);
        }
    }

    void push(uint32_t w0, uint32_t w1) { code[run].push_back(SbInsn{w0, w1}); }

    void consume(int id) {
        Node& n = nodes[id];
        if (--n.pending == 0 && n.slot >= 0) { slot_busy[(size_t)n.slot] = 0; n.slot = -1; }
    }

    void park(int id) {
        const int s = alloc_slot();
        nodes[id].slot = s;
        push(sb_w0(SB_CASE_STORE, 0, (unsigned)s), 0);
    }

    /* Index of a source constant: bank slots, then the program's affine entries, then its literals. */
    unsigned source_index(const Node& n) {
        if (n.type == N_BANK) return n.index;
        if (n.type == N_AFFINE) return (unsigned)rules.num_constants + n.index;
        float f;
        std::memcpy(&f, &n.bits, 4);
        size_t i = lit_base;
        for (; i < out.lits.size(); ++i)
            if (!std::memcmp(&out.lits[i], &f, 4)) break;
        if (i == out.lits.size()) out.lits.push_back(f);
        return (unsigned)(rules.num_constants + n_affine + (i - lit_base));
    }

    /* Constant-table entry holding a constant leaf (or a toggle among constant leaves): appends
     * "load it; store entry" to the bank part the first time the leaf is needed. */
    int entry_for(int id) {
        Node& n = nodes[id];
        if (n.entry >= 0) return n.entry;
        if (n.type != N_TOGGLE) {
            const uint32_t key = n.type == N_LIT ? n.bits : n.index;
            for (const LeafEntry& l : leaf_entries)
                if (l.type == n.type && l.key == key) return nodes[id].entry = l.entry;
        }
        const Run saved = run;
        run = RUN_BANK;
        emit_reading(SB_CASE_LOAD, id);
        const int e = (int)n_entries++;
        push(sb_w0(SB_CASE_STOREH, 0, (unsigned)e), 0);
        run = saved;
        nodes[id].entry = e;
        if (nodes[id].type != N_TOGGLE) leaf_entries.push_back(LeafEntry{nodes[id].type, nodes[id].type == N_LIT ? nodes[id].bits : nodes[id].index, e});
        return e;
    }

    /* Descriptor of a parked or hoisted node or of a direct (non-toggle) leaf, in the run being emitted. */
    Operand describe(int id) {
        const Node& n = nodes[id];
        if (n.slot >= 0) return Operand{SB_KIND_SLOT, (unsigned)n.slot};
        if (n.hoisted >= 0 && run != RUN_BANK) return Operand{SB_KIND_ROW, SB_ROW_HOISTED | (unsigned)n.hoisted};
        if (n.entry >= 0) return Operand{run == RUN_BANK ? (unsigned)SB_KIND_ROW : (unsigned)SB_KIND_CST, (unsigned)n.entry};
        if (n.type == N_COL) return rules.columns_are_slots ? Operand{SB_KIND_SLOT, n.index} : Operand{SB_KIND_ROW, n.index};
        if (!rules.split_parts || run == RUN_BANK) return Operand{SB_KIND_CST, source_index(n)};
        return Operand{SB_KIND_CST, (unsigned)entry_for(id)};
    }

    /* Emits instruction "case_base + kind(operand)" reading `id`; an unparked toggle turns the
     * instruction into a patch site with one alternative per selectable leaf.  Does not consume. */
    void emit_reading(unsigned case_base, int id) {
        const Node& n = nodes[id];
        const bool open_toggle = n.type == N_TOGGLE && n.slot < 0 && n.entry < 0;
        if (open_toggle && rules.split_parts && run != RUN_BANK && n.cls <= VC_BANK) {
            /* a toggle among constants is resolved once per bank in the bank part */
            const int e = entry_for(id);
            push(sb_w0(case_base + SB_KIND_CST, 0, (unsigned)e), 0);
            return;
        }
        if (open_toggle) {
            SbPatch p;
            std::memset(&p, 0, sizeof(p));
            p.bit0 = n.bit0;
            p.bit1 = n.bit1;
            for (unsigned i = 0; i < 4; ++i) { /* describing a constant leaf may append to the bank part first */
                const Operand o = describe(nodes[id].child[i < nodes[id].ways ? i : 0]);
                p.alt[i] = SbInsn{sb_w0(case_base + o.kind, 0, o.index), 0};
            }
            p.insn = (uint16_t)code[run].size();
            if (code[run].size() > 0xffffu) error = SECANT_ERROR_REGISTER_OVERFLOW;
            /* a site of the bank part names itself in the second word (1 + its position among the
             * program's sites, which begin with the bank part's): the scalar machine serves several
             * permutations at once and lets every lane take its own alternative */
            if (run == RUN_BANK)
                for (unsigned i = 0; i < 4; ++i) p.alt[i].w1 = (uint32_t)sites[RUN_BANK].size() + 1u;
            sites[run].push_back(p);
            push(p.alt[0].w0, p.alt[0].w1);
        } else {
            const Operand o = describe(id);
            push(sb_w0(case_base + o.kind, 0, o.index), 0);
        }
    }

    static unsigned reversed(unsigned op) {
        if (op == SB_BIN_SUB) return SB_BIN_RSUB;
        if (op == SB_BIN_DIV) return SB_BIN_RDIV;
        return op;
    }
    static unsigned bin_case(unsigned op) { return SB_CASE_BIN + op * SB_NUM_KINDS; }

    void gen(int id) {
        if (error != SECANT_SUCCESS) return;
        if (ready(id)) { emit_reading(SB_CASE_LOAD, id); return; }
        const NodeType type = nodes[id].type; /* copies: the vector may grow below */
        const unsigned op = nodes[id].op;
        if (type == N_UN) {
            const int child = nodes[id].child[0];
            gen(child);
            push(sb_w0(SB_CASE_UN + op, 0, 0), 0);
            consume(child);
        } else if (type == N_BIN) {
            const int l = nodes[id].child[0], r = nodes[id].child[1];
            if (l == r || ready(r)) {          /* acc = l ; acc = acc op r (l == r: gen parks it first) */
                gen(l);
                emit_reading(bin_case(op), r);
            } else if (ready(l)) {             /* acc = r ; acc = l op acc */
                gen(r);
                emit_reading(bin_case(reversed(op)), l);
            } else {                           /* both computed: the hungrier one goes through a slot */
                const bool left_first = nodes[l].su >= nodes[r].su;
                const int first = left_first ? l : r, second = left_first ? r : l;
                gen(first);
                if (nodes[first].slot < 0) park(first);
                gen(second);
                emit_reading(bin_case(left_first ? reversed(op) : op), first);
            }
            consume(l);
            consume(r);
        } else {
            gen_fma(Node(nodes[id]));
        }
        if (nodes[id].uses > 1) park(id);
    }

    void gen_fma(const Node& n) {
        int ch[3] = {n.child[0], n.child[1], n.child[2]};
        if (run != RUN_BANK) uses_scratch = true;
        /* a toggle operand (selected by a patched LOAD) or a hoisted per-row value cannot be
         * named by the FMA instruction: load it and park it in a private slot */
        for (int i = 0; i < 3; ++i) {
            const int id = ch[i];
            const bool toggle = nodes[id].type == N_TOGGLE && nodes[id].slot < 0 && nodes[id].entry < 0;
            const bool hrow = nodes[id].hoisted >= 0 && nodes[id].slot < 0 && run != RUN_BANK;
            const bool table = run == RUN_BANK && nodes[id].entry >= 0 && nodes[id].slot < 0;
            if (!toggle && !hrow && !table) continue;
            emit_reading(SB_CASE_LOAD, id);
            nodes.emplace_back();
            nodes.back().type = N_UN;
            nodes.back().cls = VC_MIXED;
            const int temp = (int)nodes.size() - 1;
            mem.touched.push_back(temp);
            park(temp);
            for (int j = i; j < 3; ++j)
                if (ch[j] == id) { ch[j] = temp; ++nodes[temp].uses; ++nodes[temp].pending; consume(id); }
        }
        int todo[3], cnt = 0;
        for (int i = 0; i < 3; ++i) {
            bool seen = false;
            for (int j = 0; j < i; ++j) seen = seen || ch[j] == ch[i];
            if (!seen && !ready(ch[i])) todo[cnt++] = ch[i];
        }
        for (int i = 0; i < cnt; ++i)
            for (int j = i + 1; j < cnt; ++j)
                if (nodes[todo[j]].su > nodes[todo[i]].su) std::swap(todo[i], todo[j]);
        int in_acc = -1;
        for (int i = 0; i < cnt; ++i) {
            gen(todo[i]);
            if (nodes[todo[i]].slot >= 0) continue;     /* shared: gen parked it already */
            int positions = 0;
            for (int j = 0; j < 3; ++j) positions += ch[j] == todo[i];
            if (i + 1 < cnt || positions > 1) park(todo[i]);
            else in_acc = todo[i];
        }
        unsigned kinds = 0, idx = 0;
        for (int i = 0; i < 3; ++i) {
            unsigned kind = SB_FMA_ACC, index = 0;
            if (ch[i] != in_acc) {
                const Operand o = describe(ch[i]);
                kind = o.kind;
                index = o.index;
            }
            if (index >= 512u) { error = SECANT_ERROR_REGISTER_OVERFLOW; index = 0; }
            kinds |= kind << (2 * i);
            idx |= index << (10 * i);
        }
        push(sb_w0(SB_CASE_FMA, kinds, 0), idx);
        for (int i = 0; i < 3; ++i) consume(ch[i]);
    }

    /* Computes node `id` in run `r` and leaves it where later runs can read it. */
    void hoist(Run r, int id) {
        begin_phase(r, id);
        gen(id);
        if (error != SECANT_SUCCESS) return;
        if (r == RUN_BANK) {
            const unsigned e = n_entries++;
            push(sb_w0(SB_CASE_STOREH, 0, e), 0);
            nodes[id].entry = (int32_t)e;
        } else {
            const unsigned h = n_hoisted++;
            push(sb_w0(SB_CASE_STOREH, 0, h), 0);
            nodes[id].hoisted = (int32_t)h;
        }
    }
};

}  // namespace

ProgramRules rollout_rules(size_t num_states, size_t num_constants, unsigned toggle_bits) {
    ProgramRules rules;
    rules.num_columns = num_states;
    rules.num_constants = num_constants;
    rules.banks_allowed = true;
    rules.toggle_bits = toggle_bits;
    rules.columns_are_slots = true;
    rules.reserved_slots = (unsigned)num_states;
    rules.split_parts = true;
    rules.hoist_bank = true;
    rules.fuse_store_load = true;
    return rules;
}

SecantResult routine_arities(const SecantAstProgramList& routines, uint8_t* arity) {
    if (routines.count > SECANT_AST_MAX_ROUTINES || (routines.count && !routines.items)) return SECANT_ERROR_INVALID_VALUE;
    for (size_t i = 0; i < routines.count; ++i) {
        const SecantAstInstruction* code = routines.items[i];
        unsigned count = 0;
        size_t at = 0, n = 0;
        bool done = false;
        if (!code) return SECANT_ERROR_ROUTINE_IDX_OUT_OF_BOUNDS;
        for (; n < SECANT_AST_MAX_PROGRAM_INSTRUCTIONS && !done; ++n) {
            const SecantAstInstruction* ins = code + at;
            const size_t width = secant_ast_instruction_size_get(ins);
            if (!width) return SECANT_ERROR_BAD_PROGRAM;
            if (ins[0] == SECANT_AST_INSTRUCTION_TYPE_ROUTINE_ARG_F32) {
                if (ins[1] >= SECANT_AST_MAX_INSTRUCTION_ARGS) return SECANT_ERROR_TOO_MANY_ARGS;
                if (ins[1] + 1u > count) count = ins[1] + 1u;
            }
            done = ins[0] == SECANT_AST_INSTRUCTION_TYPE_RETURN_F32;
            at += width;
        }
        if (!done) return SECANT_ERROR_BAD_PROGRAM;
        arity[i] = (uint8_t)count;
    }
    return SECANT_SUCCESS;
}

/* Token-level scan of one program up to its RETURN: the checks of read_token() plus the one rule
 * that needs context, a toggle must directly follow as many direct leaves as it selects among. */
SecantResult preflight(const SecantAstInstruction* program, const ProgramRules& rules) {
    if (!program) return SECANT_ERROR_BAD_PROGRAM;
    size_t leaves_in_a_row = 0;
    const SecantAstInstruction* ins = program;
    for (size_t n = 0; n < SECANT_AST_MAX_PROGRAM_INSTRUCTIONS; ++n) {
        Token t;
        const SecantResult status = read_token(ins, rules, &t);
        if (status != SECANT_SUCCESS) return status;
        if (t.kind == TK_RETURN) return SECANT_SUCCESS;
        if (t.kind == TK_TOGGLE && leaves_in_a_row < t.ways) return SECANT_ERROR_BAD_PROGRAM;
        leaves_in_a_row = direct_leaf(t.kind) ? leaves_in_a_row + 1 : 0;
        ins += t.width;
    }
    return SECANT_ERROR_BAD_PROGRAM;
}

SecantResult encode_program(const SecantAstInstruction* program, const SecantAstProgramList& routines,
                            const uint8_t* routine_arity, const ProgramRules& rules, EncodedBatch& out) {
    static thread_local Scratch mem;
    mem.begin();
    std::vector<Node>& nodes = mem.nodes;
    std::vector<SbAffine>& affines = mem.affines;
    Parser parser{routines, routine_arity, rules, nodes, affines};
    int root = -1;
    SecantResult r = parser.frame(program, nullptr, 0, 0, &root);
    if (r != SECANT_SUCCESS) return r;

    SbProgram rec;
    std::memset(&rec, 0, sizeof(rec));
    rec.insn_off = (uint32_t)out.insns.size();
    rec.patch_off = (uint32_t)out.patches.size();
    rec.affine_off = (uint32_t)out.affines.size();
    rec.lit_off = (uint32_t)out.lits.size();

    Emitter em(mem, rules, out);
    em.slots_high = rules.reserved_slots;
    const ValueClass root_class = nodes[root].cls;
    if (rules.split_parts) { /* rollout records (columns_are_slots) have no row-only class: only bank roots turn up */
        if ((rules.hoist_bank && parser.of_class[VC_LITERAL] + parser.of_class[VC_BANK]) || (rules.hoist_row && parser.of_class[VC_ROW]))
            em.collect(root, false, mem.bank_roots, mem.row_roots); /* otherwise there is nothing to find */
        /* row-only expressions a toggle reaches change with the permutation; what lies below them and
         * does not is worth a value of its own, computed once for all permutations of an item */
        std::vector<int>& chosen = mem.chosen;
        for (int id : mem.row_roots) {
            if (nodes[id].toggled) {
                if (rules.hoist_toggled) chosen.push_back(id);
                em.collect_shared(id, mem.shared_roots);
            } else {
                mem.shared_roots.push_back(id);
            }
        }
        /* keep the costliest values when there are more than the kernel has room for */
        chosen.insert(chosen.begin(), mem.shared_roots.begin(), mem.shared_roots.end());
        if (chosen.size() > rules.max_hoisted) {
            for (size_t i = 1; i < chosen.size(); ++i) { /* a few values: by insertion, equal weights in their order */
                const int id = chosen[i];
                size_t k = i;
                for (; k && nodes[chosen[k - 1]].weight < nodes[id].weight; --k) chosen[k] = chosen[k - 1];
                chosen[k] = id;
            }
            chosen.resize(rules.max_hoisted);
        }
        /* operands before the expressions that use them: children were created first */
        std::sort(mem.bank_roots.begin(), mem.bank_roots.end());
        std::sort(chosen.begin(), chosen.end());
        for (int id : mem.bank_roots) em.hoist(RUN_BANK, id);
        for (int id : chosen)
            if (!nodes[id].toggled) em.hoist(RUN_SHARED, id);
        for (int id : chosen)
            if (nodes[id].toggled) em.hoist(RUN_ROW, id);
        if (em.error != SECANT_SUCCESS) return em.error;
    }
    em.begin_phase(RUN_MAIN, root); /* counts the RETURN as the root's first use */
    em.gen(root);
    if (em.error != SECANT_SUCCESS) return em.error;
    em.consume(root);

    if (rules.fuse_store_load) { /* a toggle site keeps its own instruction: its alternatives are whole instructions */
        std::vector<SbInsn>& code = em.code[RUN_MAIN];
        std::vector<uint8_t>& is_site = mem.is_site;
        is_site.assign(code.size(), 0);
        for (const SbPatch& p : em.sites[RUN_MAIN]) is_site[p.insn] = 1;
        std::vector<SbInsn>& fused = mem.fused;
        std::vector<uint32_t>& moved = mem.moved;
        fused.clear();
        moved.assign(code.size(), 0);
        for (size_t i = 0; i < code.size(); ++i) {
            const unsigned cs = code[i].w0 & 0xffu;
            moved[i] = (uint32_t)fused.size();
            if (cs == SB_CASE_STORE && i + 1 < code.size() && !is_site[i + 1]) {
                const unsigned next = code[i + 1].w0 & 0xffu;
                if (next >= SB_CASE_LOAD && next < SB_CASE_LOAD + SB_NUM_KINDS) {
                    SbInsn both = code[i];
                    both.w1 = SB_STORE_THEN_LOAD | ((uint32_t)(next - SB_CASE_LOAD) << 16) | (code[i + 1].w0 >> 16);
                    fused.push_back(both);
                    moved[i + 1] = moved[i]; /* a site never sits on the absorbed load */
                    ++i;
                    continue;
                }
            }
            fused.push_back(code[i]);
        }
        for (SbPatch& p : em.sites[RUN_MAIN]) p.insn = (uint16_t)moved[p.insn];
        code.swap(fused);
    }

    /* assemble: bank part | shared row prelude | row prelude | main part, each closed by END; patch
     * sites become positions inside the whole record */
    size_t offset[NUM_RUNS] = {0, 0, 0, 0}, total = 0;
    for (int k = 0; k < NUM_RUNS; ++k) {
        offset[k] = total;
        if (k == RUN_MAIN || !em.code[k].empty()) total += em.code[k].size() + 1;
    }
    uint64_t cost = 0, pre_cost = 0;
    for (const SbInsn& i : em.code[RUN_MAIN]) cost += (uint64_t)insn_weight(i);
    for (const SbInsn& i : em.code[RUN_SHARED]) pre_cost += (uint64_t)insn_weight(i);
    for (const SbInsn& i : em.code[RUN_ROW]) pre_cost += (uint64_t)insn_weight(i);
    for (int k = 0; k < NUM_RUNS; ++k) {
        if (k != RUN_MAIN && em.code[k].empty()) continue;
        out.insns.insert(out.insns.end(), em.code[k].begin(), em.code[k].end());
        out.insns.push_back(SbInsn{sb_w0(SB_CASE_END, 0, 0), 0});
        for (SbPatch p : em.sites[k]) {
            const size_t at = offset[k] + p.insn;
            if (at > 0xffffu) return SECANT_ERROR_REGISTER_OVERFLOW;
            p.insn = (uint16_t)at;
            out.patches.push_back(p);
        }
    }

    const size_t n_patch = out.patches.size() - rec.patch_off;
    const size_t n_lits = out.lits.size() - rec.lit_off;
    if (total > 0xffffu || n_patch > 0xffffu || affines.size() + n_lits + rules.num_constants > 511u || em.n_entries > 511u ||
        em.n_hoisted > 255u)
        return SECANT_ERROR_REGISTER_OVERFLOW;
    out.affines.insert(out.affines.end(), affines.begin(), affines.end());
    if (n_patch) {
        const auto each_bit = [&](auto&& f) {
            for (size_t i = rec.patch_off; i < out.patches.size(); ++i) {
                f(out.patches[i].bit0);
                if (out.patches[i].bit1 != 0xff) f(out.patches[i].bit1);
            }
        };
        each_bit([&](uint8_t& b) { rec.bit_mask |= 1u << b; });
        if (rules.number_bits) each_bit([&](uint8_t& b) { b = (uint8_t)__builtin_popcount(rec.bit_mask & ((1u << b) - 1u)); });
        if (rules.number_bits) rec.bits = (uint16_t)__builtin_popcount(rec.bit_mask);
    }
    rec.n_insn = (uint16_t)total;
    rec.n_patch = (uint16_t)n_patch;
    rec.n_affine = (uint16_t)affines.size();
    rec.n_lits = (uint16_t)n_lits;
    rec.n_slots = (uint16_t)em.slots_high;
    rec.n_ops = (uint16_t)(parser.n_ops > 0xffffu ? 0xffffu : parser.n_ops);
    rec.pre_off = (uint16_t)offset[RUN_SHARED];
    rec.mid_off = (uint16_t)offset[RUN_ROW];
    rec.main_off = (uint16_t)offset[RUN_MAIN];
    rec.n_hoisted = (uint16_t)em.n_hoisted;
    rec.n_cst = (uint16_t)em.n_entries;
    rec.n_btmp = (uint16_t)em.btmp_high;
    const bool bank_independent = rules.split_parts && !rules.columns_are_slots && (root_class == VC_LITERAL || root_class == VC_ROW);
    rec.flags = (uint16_t)((bank_independent ? SB_PROG_BANK_INDEPENDENT : 0) | (em.uses_scratch ? SB_PROG_USES_SCRATCH : 0));
    /* cost of one row pass: the main part (plus the loss epilogue) per bank group, the prelude once;
     * the kernel scales the first term by the bank groups an item covers */
    rec.cost = (uint32_t)std::min<uint64_t>(0xffffu, cost + 6) | ((uint32_t)std::min<uint64_t>(0xffffu, pre_cost) << 16);
    out.programs.push_back(rec);
    out.max_insn = std::max<unsigned>(out.max_insn, (unsigned)total);
    out.max_extra = std::max<unsigned>(out.max_extra, (unsigned)(affines.size() + n_lits));
    out.max_slots = std::max(out.max_slots, em.slots_high);
    out.max_patch = std::max<unsigned>(out.max_patch, (unsigned)n_patch);
    out.max_hoisted = std::max(out.max_hoisted, em.n_hoisted);
    out.max_cst = std::max(out.max_cst, em.n_entries);
    out.max_btmp = std::max(out.max_btmp, em.btmp_high);
    out.uses_scratch = out.uses_scratch || em.uses_scratch;
    return SECANT_SUCCESS;
}

}  // namespace sb
