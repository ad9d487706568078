/*
 * runner.cpp - the blocking bulk runner: validate, clear, encode -> upload -> evaluate.
 *
 * Mirrors the reference runner's contract (projects/secant/s_cubin_runner.c:243-352,
 * s_runner_pipeline.c:320-427) with a different pipeline underneath.  The reference
 * specializes machine code on worker threads, loads one CUDA module per program batch,
 * launches it, waits and unloads it, so the GPU idles between modules.  Here worker
 * threads encode program batches into records, the calling thread copies each batch to
 * the device through pinned memory on a copy stream, and the resident evaluator kernel
 * of batch k runs while batch k+1 is being encoded and uploaded.  Nothing is loaded or
 * unloaded, so the "module" counters of the statistics count program batches.
 *
 * A batch is encoded in pieces of 16 to 128 programs which the workers and the calling thread take
 * in order, so the first launch of a call waits for its batch divided by the threads, not for one
 * thread that encodes all of it (2,048 programs of 32 tokens: 7.3 ms before the first launch with
 * one thread per batch, see kPiece below for the sizes).
 */
#include "evaluator.cuh"
#include "internal.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

/* Fault hooks: in the host-only test build (Makefile target `fakecuda`) the named sites ask the test
 * harness whether to fail; in the product they compile to nothing. */
#ifdef SECANT_B200_FAULT_HOOKS
extern "C" int secant_b200_fault_hook(const char* site);
#define SB_FAULT(site) (secant_b200_fault_hook(site) != 0)
#else
#define SB_FAULT(site) false
#endif

namespace sb {

std::atomic<uint64_t> g_kernel_launches{0};
std::atomic<uint64_t> g_row_stream_bytes{0};
void note_kernel_launches(unsigned n) { g_kernel_launches.fetch_add(n); }

/* cuCtxGetCurrent without linking the driver library: the library must load on machines
 * that have no GPU driver at all. */
void* current_context(bool* ok) {
    typedef int (*GetCurrentFn)(void**);
    static const GetCurrentFn fn = [] {
        void* entry = nullptr;
        cudaDriverEntryPointQueryResult status;
        return cudaGetDriverEntryPoint("cuCtxGetCurrent", &entry, cudaEnableDefault, &status) == cudaSuccess &&
                       status == cudaDriverEntryPointSuccess
                   ? reinterpret_cast<GetCurrentFn>(entry) : nullptr;
    }();
    void* ctx = nullptr;
    *ok = fn && fn(&ctx) == 0;
    return ctx;
}

namespace {

double now_seconds() {
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

/* Programs per piece: enough pieces that the last ones do not leave threads idle, none so small that
 * taking it costs as much as encoding it (a program takes about 2 us, a hand-over under 1 us). */
constexpr size_t kPieceMin = 16, kPieceMax = 128, kPiecesPerThread = 4;
constexpr size_t kMinBatch = 4096; /* programs of a batch, when the run has as many */
constexpr size_t kGramFloats = (size_t)1 << 24; /* predictions of a range of rows, see launch_gram_batch() */
constexpr size_t kSlots = 3; /* batches encoded, uploaded or running at a time */

struct Piece {
    EncodedBatch enc;
    SecantResult status = SECANT_SUCCESS;
};

/* Where the sections of a batch's records begin: programs | insns | patches | affines | lits, in bytes. */
struct Sections {
    size_t insn = 0, patch = 0, affine = 0, lit = 0, total = 0;
    Sections() = default;
    Sections(size_t programs, size_t insns, size_t patches, size_t affines, size_t lits) {
        insn = align256(programs * sizeof(SbProgram));
        patch = align256(insn + insns * sizeof(SbInsn));
        affine = align256(patch + patches * sizeof(SbPatch));
        lit = align256(affine + affines * sizeof(SbAffine));
        total = align256(lit + lits * sizeof(float) + 16);
    }
};
struct Counts { size_t insn = 0, patch = 0, affine = 0, lit = 0; };

struct Slot {
    std::vector<Piece> pieces;
    size_t used_pieces = 0;         /* of the batch held */
    size_t programs = 0;            /* of the batch held */
    /* Whoever encodes a piece also puts it where the upload takes it from, while it is in that processor's cache
     * and the others still encode: the calling thread alone needed 220 us for 3,000 programs.  Sections have room by
     * what the batch before had (`usual`, per program); where that is not enough the calling thread packs the batch. */
    bool packing = false;
    Sections place;
    Counts room, taken;             /* elements of each section; `taken` is guarded by the runner's mutex */
    double usual[4] = {0, 0, 0, 0};
    size_t done_pieces = 0;         /* encoded, guarded by the runner's mutex */
    std::vector<uint64_t> order, order_tmp; /* launch order of the batch's programs, see order_programs() */
    std::vector<SbProgram> headers;
    void* pinned = nullptr;
    size_t pinned_cap = 0;
    void* device = nullptr;
    size_t device_cap = 0;
    cudaEvent_t uploaded = nullptr;
    std::vector<cudaEvent_t> done;  /* one per compute stream */
    std::vector<char> used;         /* which compute streams this batch touched */
};

/* Programs of an uploaded batch that are launched together: its programs from `first` on, in launch order. */
struct View {
    DeviceBatch batch;
    size_t first;
    RowCut rules[2] = {}; /* of a joint view: how its two kinds' rows are cut when they are launched apart */
};

}  // namespace
}  // namespace sb

using namespace sb;

constexpr size_t kDefaultScratchFloats = (size_t)1 << 28; /* 1 GiB of scratch per launch: partial sums or predictions, and constant tables */

struct SecantCubinRunnerImpl {
    SecantCubinPlan owned_plan;     /* used when created straight from a recipe */
    const SecantCubinPlan* plan = nullptr;
    void* context = nullptr;
    int device = 0, sm_count = 0;
    size_t smem_limit = 0;
    std::vector<cudaStream_t> streams;
    std::vector<void*> scratch;      /* per compute stream: partial sums (or predictions) and constant tables of the launch in flight */
    std::vector<size_t> scratch_cap;
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t ev_join = nullptr, ev_start = nullptr, ev_stop = nullptr;
    std::vector<Slot> slots;
    std::vector<std::thread> workers;
    std::vector<double> worker_seconds;
    std::mutex mutex;
    std::condition_variable cv_work, cv_ready;
    /* current job, guarded by mutex */
    bool job_active = false;
    const SecantAstProgramSet* job_programs = nullptr;
    const uint8_t* job_arity = nullptr;
    ProgramRules job_rules;
    size_t job_batch_size = 0, job_piece_size = 0, job_pieces_per_batch = 0, job_num_pieces = 0, job_next_piece = 0;
    size_t job_open_batches = 0;   /* batches whose slot is free to be encoded into */
    size_t job_encoding = 0;       /* pieces being encoded */
    double job_encode_seconds = 0; /* summed over the pieces */
    bool job_abort = false;
    /* handle state */
    bool active = false, failed = false, shutdown = false;
    size_t populations = 0;        /* device-resident populations created from this runner and not yet destroyed */
    size_t scratch_limit = kDefaultScratchFloats; /* secant_b200_runner_set_scratch_limit */
    uint32_t fast_math = 0;        /* secant_b200_runner_set_math */
    std::string last_error;
};


/* A population kept on the device: programs validated, encoded and uploaded once, then
 * scored any number of times (new data, new coefficient banks) without touching the host
 * copies again. */
struct SecantB200PopulationImpl {
    SecantCubinRunnerImpl* runner = nullptr;
    std::vector<uint8_t> ast_bytes, routine_bytes;
    std::vector<const uint8_t*> ast_ptrs, routine_ptrs;
    SecantAstProgramSet set{};
    unsigned toggle_bits = 0;
    struct Resident { void* device = nullptr; std::vector<View> views; std::vector<SbProgram> headers; /* in launch order */ };
    std::vector<Resident> batches;
    uint64_t total_ops = 0;
};

namespace {

/* Takes the next piece of the job in order, SIZE_MAX when there is none to be had now; the caller
 * holds the mutex. */
size_t take_piece(SecantCubinRunnerImpl* r) {
    if (!r->job_active || r->job_abort || r->job_next_piece >= r->job_num_pieces) return SIZE_MAX;
    if (r->job_next_piece / r->job_pieces_per_batch >= r->job_open_batches) return SIZE_MAX;
    ++r->job_encoding;
    return r->job_next_piece++;
}

/* Copies a piece's arrays to the slot's pinned buffer, from the elements `at` of its sections on, and its headers (whose
 * offsets move by that) to the batch's programs from `program` on. */
void pack_piece(Slot& s, const Sections& place, const EncodedBatch& e, const Counts& at, size_t program) {
    char* const h = static_cast<char*>(s.pinned);
    SbProgram* out = s.headers.data() + program;
    for (SbProgram p : e.programs) {
        p.insn_off += (uint32_t)at.insn; p.patch_off += (uint32_t)at.patch;
        p.affine_off += (uint32_t)at.affine; p.lit_off += (uint32_t)at.lit;
        *out++ = p;
    }
    if (!e.insns.empty()) std::memcpy(h + place.insn + at.insn * sizeof(SbInsn), e.insns.data(), e.insns.size() * sizeof(SbInsn));
    if (!e.patches.empty()) std::memcpy(h + place.patch + at.patch * sizeof(SbPatch), e.patches.data(), e.patches.size() * sizeof(SbPatch));
    if (!e.affines.empty()) std::memcpy(h + place.affine + at.affine * sizeof(SbAffine), e.affines.data(), e.affines.size() * sizeof(SbAffine));
    if (!e.lits.empty()) std::memcpy(h + place.lit + at.lit * sizeof(float), e.lits.data(), e.lits.size() * sizeof(float));
}

/* Makes a slot ready for a batch: room for its headers, and for its records where the slot's buffers are large enough
 * for what they usually take.  The caller holds the mutex or no job runs on the slot. */
void prepare_slot(Slot& s, size_t programs) {
    s.programs = programs;
    s.headers.resize(programs);
    s.taken = Counts();
    const auto room = [&](int k) { return (size_t)(s.usual[k] * 1.15 * (double)programs) + 128; };
    s.room.insn = room(0); s.room.patch = room(1); s.room.affine = room(2); s.room.lit = room(3);
    s.place = Sections(programs, s.room.insn, s.room.patch, s.room.affine, s.room.lit);
    s.packing = s.usual[0] > 0 && s.place.total <= s.pinned_cap && s.place.total <= s.device_cap && s.place.total < (size_t)1 << 32;
}

/* Encodes piece `index` into its slot; `lock` (held) is released meanwhile. */
void encode_piece(SecantCubinRunnerImpl* r, std::unique_lock<std::mutex>& lock, size_t index, double* seconds) {
    const SecantAstProgramSet* programs = r->job_programs;
    const uint8_t* arity = r->job_arity;
    const ProgramRules rules = r->job_rules;
    const size_t batch = index / r->job_pieces_per_batch, within = index % r->job_pieces_per_batch;
    Slot& slot = r->slots[batch % r->slots.size()];
    Piece& piece = slot.pieces[within];
    const size_t batch_first = batch * r->job_batch_size;
    const size_t batch_end = std::min(programs->asts.count, batch_first + r->job_batch_size);
    const size_t first = batch_first + within * r->job_piece_size;
    const size_t end = std::min(batch_end, first + r->job_piece_size);
    lock.unlock();

    const double begin = now_seconds();
    SecantResult status = SECANT_SUCCESS;
    try { /* an allocation failure inside the encoder must reach the caller as a result code */
        piece.enc.clear();
        for (size_t i = first; i < end && status == SECANT_SUCCESS; ++i) {
            status = encode_program(programs->asts.items[i], programs->routines, arity, rules, piece.enc);
            if (status == SECANT_SUCCESS) piece.enc.programs.back().index = (uint32_t)i;
        }
    } catch (...) {
        status = SECANT_ERROR_ALLOCATION_FAILED;
    }
    if (SB_FAULT("encode")) status = SECANT_ERROR_BAD_PROGRAM;
    if (status == SECANT_SUCCESS && slot.packing) {
        Counts at;
        const EncodedBatch& e = piece.enc;
        lock.lock();
        at = slot.taken;
        slot.taken.insn += e.insns.size(); slot.taken.patch += e.patches.size(); slot.taken.affine += e.affines.size(); slot.taken.lit += e.lits.size();
        lock.unlock();
        if (at.insn + e.insns.size() <= slot.room.insn && at.patch + e.patches.size() <= slot.room.patch &&
            at.affine + e.affines.size() <= slot.room.affine && at.lit + e.lits.size() <= slot.room.lit)
            pack_piece(slot, slot.place, e, at, first - batch_first);
    }
    const double spent = now_seconds() - begin;

    lock.lock();
    piece.status = status;
    *seconds += spent;
    r->job_encode_seconds += spent;
    --r->job_encoding;
    if (++slot.done_pieces == slot.used_pieces || r->job_abort) r->cv_ready.notify_all();
}

void worker_main(SecantCubinRunnerImpl* r, size_t worker_index) {
    std::unique_lock<std::mutex> lock(r->mutex);
    for (;;) {
        size_t piece = SIZE_MAX;
        r->cv_work.wait(lock, [&] { return r->shutdown || (piece = take_piece(r)) != SIZE_MAX; });
        if (r->shutdown) return; /* no job is active then */
        encode_piece(r, lock, piece, &r->worker_seconds[worker_index]);
    }
}

SecantResult cuda_fail(SecantCubinRunnerImpl* r, cudaError_t e, const char* what) {
    char text[256];
    std::snprintf(text, sizeof(text), "%s: %s", what, cudaGetErrorString(e));
    r->last_error = text;
    return SECANT_ERROR_DRIVER_FAILED;
}
#define SB_CUDA(call, what) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) return cuda_fail(r, e_, what); } while (0)

SecantResult runner_init(SecantCubinRunnerImpl* r, const SecantCubinRunnerOptions* options) {
    bool ok = false;
    SB_CUDA(cudaGetDevice(&r->device), "cudaGetDevice");
    SB_CUDA(cudaFree(nullptr), "context initialisation");
    r->context = current_context(&ok);
    if (!ok || !r->context) { r->last_error = "no current CUDA context"; return SECANT_ERROR_INVALID_STATE; }
    int value = 0;
    SB_CUDA(cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, r->device), "device attributes");
    r->sm_count = value;
    SB_CUDA(cudaDeviceGetAttribute(&value, cudaDevAttrMaxSharedMemoryPerBlockOptin, r->device), "device attributes");
    r->smem_limit = (size_t)value;
    SB_CUDA(configure_kernels(), "kernel attributes");
    r->streams.resize(options->num_streams);
    for (auto& s : r->streams) SB_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate");
    r->scratch.assign(r->streams.size(), nullptr);
    r->scratch_cap.assign(r->streams.size(), 0);
    SB_CUDA(cudaStreamCreateWithFlags(&r->copy_stream, cudaStreamNonBlocking), "cudaStreamCreate");
    SB_CUDA(cudaEventCreateWithFlags(&r->ev_join, cudaEventDisableTiming), "cudaEventCreate");
    SB_CUDA(cudaEventCreate(&r->ev_start), "cudaEventCreate");
    SB_CUDA(cudaEventCreate(&r->ev_stop), "cudaEventCreate");
    r->slots.resize(kSlots);
    for (auto& s : r->slots) {
        SB_CUDA(cudaEventCreateWithFlags(&s.uploaded, cudaEventDisableTiming), "cudaEventCreate");
        s.done.resize(r->streams.size());
        s.used.assign(r->streams.size(), 0);
        for (auto& e : s.done) SB_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    }
    r->worker_seconds.assign(options->num_workers + 1, 0.0); /* the calling thread's last */
    try {
        for (size_t i = 0; i < options->num_workers; ++i) {
            if (SB_FAULT("thread")) throw std::bad_alloc();
            r->workers.emplace_back(worker_main, r, i);
        }
    } catch (...) {
        r->last_error = "worker thread creation failed";
        return SECANT_ERROR_THREAD_FAILED;
    }
    return SECANT_SUCCESS;
}

/* Stops the workers, waits for the streams and releases everything the runner owns.  May be
 * called again after a failure: a resource is forgotten only once its release has succeeded, so a
 * second destroy retries what the first could not free. */
SecantResult runner_teardown(SecantCubinRunnerImpl* r) {
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        r->shutdown = true;
    }
    r->cv_work.notify_all();
    for (auto& t : r->workers)
        if (t.joinable()) t.join();
    r->workers.clear();
    SecantResult result = SECANT_SUCCESS;
    auto ok = [&](cudaError_t e) {
        if (e == cudaSuccess || e == cudaErrorCudartUnloading) return true;
        result = SECANT_ERROR_DRIVER_FAILED;
        return false;
    };
    for (auto& s : r->streams) if (s) ok(cudaStreamSynchronize(s));
    if (r->copy_stream) ok(cudaStreamSynchronize(r->copy_stream));
    if (result != SECANT_SUCCESS) return SECANT_ERROR_COMPLETION_UNKNOWN; /* nothing is released under work that may still run */
    for (auto& s : r->slots) {
        if (s.pinned && ok(cudaFreeHost(s.pinned))) { s.pinned = nullptr; s.pinned_cap = 0; }
        if (s.device && ok(cudaFree(s.device))) { s.device = nullptr; s.device_cap = 0; }
        if (s.uploaded && ok(cudaEventDestroy(s.uploaded))) s.uploaded = nullptr;
        for (auto& e : s.done) if (e && ok(cudaEventDestroy(e))) e = nullptr;
    }
    for (size_t k = 0; k < r->scratch.size(); ++k)
        if (r->scratch[k] && ok(cudaFree(r->scratch[k]))) { r->scratch[k] = nullptr; r->scratch_cap[k] = 0; }
    for (auto& s : r->streams) if (s && ok(cudaStreamDestroy(s))) s = nullptr;
    if (r->copy_stream && ok(cudaStreamDestroy(r->copy_stream))) r->copy_stream = nullptr;
    if (r->ev_join && ok(cudaEventDestroy(r->ev_join))) r->ev_join = nullptr;
    if (r->ev_start && ok(cudaEventDestroy(r->ev_start))) r->ev_start = nullptr;
    if (r->ev_stop && ok(cudaEventDestroy(r->ev_stop))) r->ev_stop = nullptr;
    return result;
}

SecantResult options_validate(const SecantCubinRunnerOptions* options) {
    if (!options || options->struct_size < sizeof(*options)) return SECANT_ERROR_INVALID_VALUE;
    if (options->version != SECANT_CUBIN_RUNNER_OPTIONS_VERSION_1) return SECANT_ERROR_UNSUPPORTED_VERSION;
    if (options->flags || options->reserved || !options->num_workers || !options->num_streams ||
        options->num_workers > 256 || options->num_streams > 1024)
        return SECANT_ERROR_INVALID_VALUE;
    return SECANT_SUCCESS;
}

SecantResult create_common(SecantCubinRunnerImpl* r, const SecantCubinRunnerOptions* options, SecantCubinRunner* out) {
    const SecantResult result = runner_init(r, options);
    if (result != SECANT_SUCCESS) {
        if (runner_teardown(r) != SECANT_SUCCESS) { /* keep ownership: destroy-only handle */
            r->failed = true;
            *out = r;
            return result;
        }
        delete r;
        return result;
    }
    *out = r;
    return SECANT_SUCCESS;
}

/* Programs whose per-warp working set (spill slots, constant table, hoisted row values) is larger
 * than this are launched separately, so that the shared-memory budget of the common case is not
 * sized by rare programs. */
constexpr unsigned kLightSlots = 2, kLightTable = 8, kLightHoisted = 4;

bool is_light(const SbProgram& p) { return p.n_slots <= kLightSlots && p.n_cst <= kLightTable && p.n_hoisted <= kLightHoisted; }

/* scheduling weight of a program: one row pass over sixteen bank groups, for every permutation of its own */
uint64_t schedule_cost(const SbProgram& p) {
    const uint64_t main_part = p.cost & 0xffffu, prelude = p.cost >> 16;
    const uint64_t once = main_part * ((p.flags & SB_PROG_BANK_INDEPENDENT) ? 1u : 16u) + prelude;
    return std::min<uint64_t>(once << std::min<unsigned>(p.bits, 32u), 0x1fffffu); /* 21 bits of the order's key */
}

/* adds what the planner weighs of a program to its batch's */
void add_weights(DeviceBatch& batch, const SbProgram& p) {
    const uint64_t cost = schedule_cost(p);
    batch.total_cost += cost;
    batch.max_cost = std::max(batch.max_cost, cost);
    batch.main_cost += p.cost & 0xffffu;
    batch.prelude_cost += p.cost >> 16;
    batch.total_perms += (double)(1ull << p.bits);
}

/* Puts the batch's programs in launch order: light programs first, heavy ones after them; inside each
 * group the costly ones first, so that every CTA, which takes a strided subset, has a queue from its
 * costliest item to its cheapest and its warps finish a tile close together; ties keep the run's order.
 * order[i] = key << 32 | position in `headers`, sorted on the 22-bit key (1 heavy bit above 21 bits of
 * inverted cost) by two counting passes. */
void order_programs(Slot& s) {
    constexpr unsigned kBits = 11, kBins = 1u << kBits;
    const size_t n = s.headers.size();
    s.order.resize(n);
    for (size_t i = 0; i < n; ++i) {
        const SbProgram& p = s.headers[i];
        const uint64_t key = (is_light(p) ? 0u : 1u << 21) | (0x1fffffu - (uint32_t)schedule_cost(p));
        s.order[i] = key << 32 | i;
    }
    if (n <= 512) { /* keys with the position below them are unique, so any sort gives the same order */
        std::sort(s.order.begin(), s.order.end());
        return;
    }
    s.order_tmp.resize(n);
    for (unsigned pass = 0; pass < 2; ++pass) {
        uint32_t at[kBins] = {0};
        const unsigned shift = 32 + pass * kBits;
        for (size_t i = 0; i < n; ++i) ++at[(s.order[i] >> shift) & (kBins - 1)];
        uint32_t sum = 0;
        for (uint32_t& a : at) { const uint32_t c = a; a = sum; sum += c; }
        for (size_t i = 0; i < n; ++i) s.order_tmp[at[(s.order[i] >> shift) & (kBins - 1)]++] = s.order[i];
        s.order.swap(s.order_tmp);
    }
}

/* Joins the batch's encoded pieces in the slot's pinned buffer (a program's offsets move by what lies
 * before its piece) unless that has been done as they were encoded, grows the buffers when needed, and enqueues the upload.
 * Layout: programs | insns | patches | affines | lits.  The pinned buffer keeps the programs' headers, in launch
 * order, until the slot is used again. */
SecantResult upload_batch(SecantCubinRunnerImpl* r, Slot& s, std::vector<View>* views) {
    const size_t n_programs = s.programs;
    Counts n;
    for (size_t q = 0; q < s.used_pieces; ++q) {
        const EncodedBatch& e = s.pieces[q].enc;
        n.insn += e.insns.size(); n.patch += e.patches.size(); n.affine += e.affines.size(); n.lit += e.lits.size();
    }
    if (n.insn > 0xffffffffull || n.patch > 0xffffffffull || n.affine > 0xffffffffull || n.lit > 0xffffffffull) return SECANT_ERROR_OVERFLOW;
    const bool packed = s.packing && n.insn <= s.room.insn && n.patch <= s.room.patch && n.affine <= s.room.affine && n.lit <= s.room.lit;
    const Sections at = packed ? s.place : Sections(n_programs, n.insn, n.patch, n.affine, n.lit);
    s.usual[0] = (double)n.insn / n_programs; s.usual[1] = (double)n.patch / n_programs;
    s.usual[2] = (double)n.affine / n_programs; s.usual[3] = (double)n.lit / n_programs;
    if (!packed) {
        const size_t total = at.total;
        if (s.pinned_cap < total) {
            if (s.pinned) SB_CUDA(cudaFreeHost(s.pinned), "cudaFreeHost");
            s.pinned = nullptr; s.pinned_cap = 0;
            SB_CUDA(cudaHostAlloc(&s.pinned, total + total / 2, cudaHostAllocDefault), "cudaHostAlloc");
            s.pinned_cap = total + total / 2;
        }
        if (s.device_cap < total) {
            if (s.device) SB_CUDA(cudaFree(s.device), "cudaFree");
            s.device = nullptr; s.device_cap = 0;
            SB_CUDA(cudaMalloc(&s.device, total + total / 2), "cudaMalloc");
            s.device_cap = total + total / 2;
        }
        Counts before;
        size_t program = 0;
        for (size_t q = 0; q < s.used_pieces; ++q) {
            const EncodedBatch& e = s.pieces[q].enc;
            pack_piece(s, at, e, before, program);
            before.insn += e.insns.size(); before.patch += e.patches.size(); before.affine += e.affines.size(); before.lit += e.lits.size();
            program += e.programs.size();
        }
    }
    const size_t o_prog = 0, o_insn = at.insn, o_patch = at.patch, o_aff = at.affine, o_lit = at.lit;
    const size_t total = align256(o_lit + n.lit * sizeof(float) + 16);
    char* h = static_cast<char*>(s.pinned);
    order_programs(s);
    SbProgram* const out = reinterpret_cast<SbProgram*>(h + o_prog);
    size_t num_light = 0;
    uint64_t entries = 0;
    for (size_t i = 0; i < n_programs; ++i) {
        out[i] = s.headers[(uint32_t)s.order[i]];
        out[i].cst_off = (uint32_t)entries;
        entries += out[i].n_cst;
        num_light += (s.order[i] >> 53) == 0;
    }
    if (entries > 0xffffffffull) return SECANT_ERROR_OVERFLOW;
    SB_CUDA(cudaMemcpyAsync(s.device, s.pinned, total, cudaMemcpyHostToDevice, r->copy_stream), "program upload");
    SB_CUDA(cudaEventRecord(s.uploaded, r->copy_stream), "cudaEventRecord");
    const char* d = static_cast<const char*>(s.device);
    views->clear();
    const size_t bounds[3] = {0, num_light, n_programs};
    for (int k = 0; k < 2; ++k) {
        if (bounds[k] == bounds[k + 1]) continue;
        DeviceBatch db;
        std::memset(&db, 0, sizeof(db));
        db.insns = reinterpret_cast<const SbInsn*>(d + o_insn);
        db.patches = reinterpret_cast<const SbPatch*>(d + o_patch);
        db.affines = reinterpret_cast<const SbAffine*>(d + o_aff);
        db.lits = reinterpret_cast<const float*>(d + o_lit);
        db.programs = reinterpret_cast<const SbProgram*>(d + o_prog) + bounds[k];
        db.num_programs = (uint32_t)(bounds[k + 1] - bounds[k]);
        db.max_insn = 1;
        for (size_t i = bounds[k]; i < bounds[k + 1]; ++i) {
            const SbProgram& p = out[i];
            db.max_insn = std::max<uint32_t>(db.max_insn, p.n_insn);
            db.max_extra = std::max<uint32_t>(db.max_extra, (uint32_t)p.n_affine + p.n_lits);
            db.max_slots = std::max<uint32_t>(db.max_slots, p.n_slots);
            db.max_hoisted = std::max<uint32_t>(db.max_hoisted, p.n_hoisted);
            db.max_cst = std::max<uint32_t>(db.max_cst, p.n_cst);
            db.total_cst += p.n_cst;
            add_weights(db, p);
            db.max_bits = std::max<uint32_t>(db.max_bits, p.bits);
            db.max_btmp = std::max<uint32_t>(db.max_btmp, p.n_btmp);
            db.uses_scratch |= (p.flags & SB_PROG_USES_SCRATCH) ? 1u : 0u;
        }
        views->push_back(View{db, bounds[k], {}});
    }
    return SECANT_SUCCESS;
}

EvalProblem make_problem(const SecantCubinPlan& plan, const UnpackedRun& run, size_t first_program) {
    EvalProblem p;
    std::memset(&p, 0, sizeof(p));
    p.input = reinterpret_cast<const float*>(run.input.address);
    p.input_ld = run.input.leading_dimension;
    p.num_inputs = (uint32_t)plan.num_inputs;
    p.targets = reinterpret_cast<const float*>(run.targets.address);
    p.targets_ld = run.targets.leading_dimension;
    p.num_targets = (uint32_t)run.num_targets;
    p.banks = reinterpret_cast<const float*>(run.banks.address);
    p.bank_stride = run.banks.bank_stride;
    p.program_bank_stride = run.program_bank_stride;
    p.first_program = first_program;
    p.num_constants = (uint32_t)plan.num_constants;
    p.num_banks = (uint32_t)run.num_banks;
    p.toggle_bits = run.toggle_bits;
    p.num_rows = run.rows;
    p.output = reinterpret_cast<float*>(run.output.address);
    switch (plan.shape) {
    case SECANT_KERNEL_SHAPE_STATIC_MATERIALIZE_F32:
        p.mode = EVAL_MATERIALIZE; p.out_program_stride = run.output.leading_dimension; p.out_target_stride = 0; break;
    case SECANT_KERNEL_SHAPE_STATIC_SSE_F32:
        p.mode = EVAL_SSE; p.out_program_stride = run.output.leading_dimension; p.out_target_stride = 1; break;
    case SECANT_KERNEL_SHAPE_STATIC_AFFINE_STATS_F32:
        p.mode = EVAL_AFFINE_STATS; p.out_program_stride = run.output.leading_dimension; p.out_target_stride = 1; break;
    case SECANT_KERNEL_SHAPE_STATIC_GRAM_STATS_F32: /* predictions are materialized into scratch; launch_gram_batch() places them */
        p.mode = EVAL_MATERIALIZE; p.output = nullptr; p.out_program_stride = 0; p.out_target_stride = 0; break;
    default:
        p.mode = EVAL_SSE;
        p.out_program_stride = run.num_targets * run.output.leading_dimension;
        p.out_target_stride = run.output.leading_dimension;
        break;
    }
    return p;
}

/* Per-stream scratch for the evaluator's per-split partial sums and constant tables.  Launches on one stream
 * run in order, so the evaluator and the kernel that folds its partial sums may reuse the buffer of the
 * launch before them; growing it waits for the stream first and takes a quarter more than is needed, as far
 * as the scratch limit allows. */
SecantResult stream_scratch(SecantCubinRunnerImpl* r, size_t k, size_t elements, float** out) {
    const size_t bytes = elements * sizeof(float);
    if (elements > SIZE_MAX / sizeof(float)) return SECANT_ERROR_OVERFLOW;
    if (r->scratch_cap[k] < bytes) {
        SB_CUDA(cudaStreamSynchronize(r->streams[k]), "cudaStreamSynchronize");
        if (r->scratch[k]) SB_CUDA(cudaFree(r->scratch[k]), "cudaFree");
        r->scratch[k] = nullptr; r->scratch_cap[k] = 0;
        const size_t most = std::max(bytes, r->scratch_limit * sizeof(float));
        const size_t want = std::min(bytes + bytes / 4, most);
        if (cudaMalloc(&r->scratch[k], want) != cudaSuccess) {
            (void)cudaGetLastError();
            r->last_error = "no device memory for the scratch of a launch";
            return SECANT_ERROR_ALLOCATION_FAILED;
        }
        r->scratch_cap[k] = want;
    }
    *out = static_cast<float*>(r->scratch[k]);
    return SECANT_SUCCESS;
}

/* The part of the machine a view's launch should count on: with two views of one run entry on two streams
 * both are on the device at a time, and when neither fills it they share it by their work. */
Neighbour view_share(const SecantCubinRunnerImpl* r, const std::vector<View>& views, const View& view, size_t entries) {
    if (r->streams.size() < 2 || entries != 1 || views.size() < 2) return Neighbour{Neighbour::NONE, 1.0};
    double all = 0.0;
    for (const View& v : views) all += (double)v.batch.total_cost;
    return Neighbour{Neighbour::SHARES, std::min(0.95, std::max(0.05, (double)view.batch.total_cost / std::max(1.0, all)))};
}

/* Half of the scratch limit is for constant tables (an entry per program constant and configuration), the rest for the
 * partial sums of the row splits, without which few programs would fill few SMs. */
bool tables_fit(const SecantCubinRunnerImpl* r, const DeviceBatch& batch, uint32_t banks) {
    return batch.total_cst <= r->scratch_limit / 2 / ((banks + 3ull) << batch.max_bits);
}

/* The programs of a view from `first` on whose constant tables take at most `most` floats, one at least.  Every
 * table of a launch has room for the permutations of the program that reads most bits, so a launch takes its
 * measure from its own programs: those with most permutations come first in launch order and mostly keep to
 * themselves (1,024 programs of which one reads 14 bits, 64 sets, 2,000 rows: 466 ms in 105 launches when the
 * largest program of the view was the measure of all). */
DeviceBatch tables_that_fit(const View& view, const SbProgram* headers, size_t first, uint32_t banks, size_t most) {
    DeviceBatch part = view.batch;
    part.programs += first;
    part.num_programs = 0;
    part.total_cst = 0;
    part.total_cost = part.max_cost = part.main_cost = part.prelude_cost = 0; /* what the planner weighs against its number of programs */
    part.total_perms = 0;
    part.max_bits = 0;
    for (size_t i = first; i < view.batch.num_programs; ++i) {
        const SbProgram& p = headers[view.first + i];
        const uint64_t entries = part.total_cst + p.n_cst;
        const uint32_t bits = std::max<uint32_t>(part.max_bits, p.bits);
        if (part.num_programs && entries > most / ((banks + 3ull) << bits)) break;
        ++part.num_programs;
        part.total_cst = entries;
        part.max_bits = bits;
        add_weights(part, p);
    }
    return part;
}

/* The views of a batch as they are launched for a run entry: light and heavy programs in one launch where that keeps
 * most of the warps, since two launches share the machine badly: the heavy programs are few, and their CTAs take an SM
 * each for an item or two, or a few SMs for long (256 resident programs, 33 sets, 10,007 rows, 14 of them heavy: 452 us
 * apart, 288 together).  Heavy programs, which are the costliest, then come first.  A grid of many waves
 * fills the machine either way, and its light programs are faster with all the warps that fit. */
std::vector<View> views_to_launch(SecantCubinRunnerImpl* r, const std::vector<View>& views, const EvalProblem& prob) {
    if (views.size() != 2 || prob.toggle_bits) return views;
    View all = views[0];
    const DeviceBatch& heavy = views[1].batch;
    DeviceBatch& b = all.batch;
    b.first = b.num_programs;
    b.num_programs += heavy.num_programs;
    b.max_insn = std::max(b.max_insn, heavy.max_insn);
    b.max_extra = std::max(b.max_extra, heavy.max_extra);
    b.max_slots = std::max(b.max_slots, heavy.max_slots);
    b.max_hoisted = std::max(b.max_hoisted, heavy.max_hoisted);
    b.max_cst = std::max(b.max_cst, heavy.max_cst);
    b.max_btmp = std::max(b.max_btmp, heavy.max_btmp);
    b.uses_scratch |= heavy.uses_scratch;
    b.total_cst += heavy.total_cst;
    b.total_cost += heavy.total_cost;
    b.max_cost = std::max(b.max_cost, heavy.max_cost);
    b.main_cost += heavy.main_cost;
    b.prelude_cost += heavy.prelude_cost;
    b.total_perms += heavy.total_perms;
    b.max_bits = std::max(b.max_bits, heavy.max_bits);
    if (!tables_fit(r, b, prob.num_banks)) return views;
    int variant = -1; /* each program's rows are added in the order of the launch its kind would have; predictions are not added */
    for (int k = 0; k < 2 && prob.mode != EVAL_MATERIALIZE; ++k) {
        const LaunchPlan alone = plan_rules(views[k].batch, prob, r->sm_count, r->smem_limit, r->scratch_limit);
        if (!alone.ok || (k && alone.variant != variant)) return views;
        variant = alone.variant;
        all.rules[k] = alone.rules[0];
    }
    const LaunchPlan plan = plan_launch(b, prob, r->sm_count, r->smem_limit, r->scratch_limit, Neighbour{Neighbour::NONE, 1.0}, all.rules);
    if (!plan.ok || (variant >= 0 && plan.variant != variant) || plan.warps < 16u || (uint64_t)plan.grid_x >= 8ull * (uint64_t)r->sm_count) return views;
    /* an item of a pass or two pays for its set-up once more when the heavy programs' memory makes the tile smaller
     * (3,000 programs without coefficients, 20,011 rows: 1 % of the call) */
    if (plan.tile_rows / (32u * (uint32_t)kVariantRows[plan.variant]) * plan.groups_per_item < 8u) {
        const LaunchPlan light = plan_launch(views[0].batch, prob, r->sm_count, r->smem_limit, r->scratch_limit);
        if (light.ok && light.tile_rows > plan.tile_rows) return views;
    }
    return {all};
}

/* Enqueues the evaluation of one device-resident batch for every run entry, spreading
 * entries over the compute streams.  `after` (optional) is an event each stream waits on
 * first; `done`/`used` (optional) receive one completion event per touched stream. */
SecantResult launch_batch(SecantCubinRunnerImpl* r, const std::vector<View>& batch_views, const SbProgram* headers,
                          const std::vector<UnpackedRun>& runs, size_t* stream_cursor, cudaEvent_t after, std::vector<cudaEvent_t>* done, std::vector<char>* used) {
    const SecantCubinPlan& plan = *r->plan;
    for (size_t e = 0; e < runs.size(); ++e) {
        EvalProblem prob = make_problem(plan, runs[e], 0); /* SbProgram::index already places every program in the run */
        prob.fast_math = r->fast_math;
        if (runs[e].program_bank_stride)
            prob.banks = reinterpret_cast<const float*>(runs[e].banks.address) + runs[e].first_program_index * runs[e].program_bank_stride;
        const std::vector<View> views = views_to_launch(r, batch_views, prob);
        /* what a view's launches should know of the last launch of the view before, on another stream; a view's own
         * launches come one after the other */
        Neighbour neighbour = view_share(r, views, views[0], runs.size());
        const bool beside = neighbour.kind != Neighbour::NONE;
        for (const View& view : views) {
        const DeviceBatch& db = view.batch;
        Neighbour next = neighbour;
        const size_t k = (*stream_cursor)++ % r->streams.size();
        cudaStream_t stream = r->streams[k];
        cudaError_t ce = after ? cudaStreamWaitEvent(stream, after, 0) : cudaSuccess;
        /* one launch, unless its constant tables would take too much: then the programs in as many launches as it
         * takes, and a program at a time at least */
        const bool whole = tables_fit(r, db, prob.num_banks);
        for (size_t first = 0; first < db.num_programs && ce == cudaSuccess;) {
            const DeviceBatch part = whole ? db : tables_that_fit(view, headers, first, prob.num_banks, r->scratch_limit / 2);
            first += part.num_programs;
            const LaunchPlan lp = plan_launch(part, prob, r->sm_count, r->smem_limit, r->scratch_limit, neighbour, part.first ? view.rules : nullptr);
            if (!lp.ok) {
                r->last_error = lp.overflow ? "configuration count beyond the evaluator's 32-bit item index" : "program batch does not fit shared memory";
                return lp.overflow ? SECANT_ERROR_OVERFLOW : SECANT_ERROR_REGISTER_OVERFLOW;
            }
            float* partial = nullptr;
            if (const size_t floats = lp.table_offset + lp.table_elements) {
                const SecantResult a = stream_scratch(r, k, floats, &partial);
                if (a != SECANT_SUCCESS) return a;
            }
            unsigned launches = 0;
            ce = launch_eval(part, prob, lp, partial, stream, &launches);
            /* the launch beside it has the SMs this one leaves; when it leaves none, the other's CTAs come behind it and are
             * best spread over all of them (2,938 programs, eleven of them heavy, 227,933 rows: 4.2 ms, 5.0 with those
             * confined to the SMs their work is worth) */
            if (beside) next = lp.grid_x < (uint32_t)r->sm_count ? Neighbour{Neighbour::LEAVES, 1.0 - (double)lp.grid_x / r->sm_count} : Neighbour{Neighbour::FILLS, 1.0};
            g_kernel_launches.fetch_add(launches);
            if (launches)
                g_row_stream_bytes.fetch_add((uint64_t)lp.num_groups * (prob.num_inputs + (prob.mode == EVAL_MATERIALIZE ? 0u : prob.num_targets)) *
                                             (uint64_t)prob.num_rows * sizeof(float));
        }
        neighbour = next;
        if (ce == cudaSuccess && done) ce = cudaEventRecord((*done)[k], stream);
        if (ce != cudaSuccess) return cuda_fail(r, ce, "kernel launch");
        if (used) (*used)[k] = 1;
        }
    }
    return SECANT_SUCCESS;
}

/* The static Gram shape: the predictions of the batch's programs are materialized for a range of
 * rows into the stream's scratch by the evaluator (every view of the batch), then reduced to the
 * cohorts' statistics, range after range on one stream, so every statistic is added to in row
 * order.  first_program is the batch's first program and a multiple of the cohort size. */
SecantResult launch_gram_batch(SecantCubinRunnerImpl* r, const std::vector<View>& batch_views, const std::vector<UnpackedRun>& runs,
                               size_t first_program, size_t batch_programs, size_t* stream_cursor, cudaEvent_t after,
                               std::vector<cudaEvent_t>* done, std::vector<char>* used) {
    const SecantCubinPlan& plan = *r->plan;
    const size_t cohort = plan.asts_per_kernel;
    for (size_t e = 0; e < runs.size(); ++e) {
        const UnpackedRun& run = runs[e];
        const size_t k = (*stream_cursor)++ % r->streams.size();
        cudaStream_t stream = r->streams[k];
        /* scratch: the range's predictions, then the constant tables of every view (padded to four banks at
         * most), which the first range makes and the others read again */
        size_t entries = 0;
        for (const View& v : batch_views) entries += v.batch.total_cst;
        /* rows per range: what the scratch limit leaves for this batch's predictions, between 128 and as many as stay in
         * L2 beside the data (64 MB) or 16,384; a multiple of four, which the kernels' loads count on */
        const size_t room = r->scratch_limit > 4 * entries ? (r->scratch_limit - 4 * entries) / 4 * 4 : 0;
        const size_t fit = room / batch_programs / 4 * 4, resident = kGramFloats / batch_programs / 4 * 4;
        const size_t range = std::min<size_t>((run.rows + 3) / 4 * 4, std::max<size_t>(128, std::min<size_t>(std::max<size_t>(16384, resident), fit)));
        EvalProblem whole = make_problem(plan, run, 0);
        whole.num_rows = range;
        const std::vector<View> views = views_to_launch(r, batch_views, whole);
        std::vector<int> tables_made(views.size(), -1); /* for which register tile */
        const size_t predictions = batch_programs * range;
        float* scratch = nullptr;
        const SecantResult a = stream_scratch(r, k, predictions + 4 * entries, &scratch);
        if (a != SECANT_SUCCESS) return a;
        cudaError_t ce = after ? cudaStreamWaitEvent(stream, after, 0) : cudaSuccess;
        for (size_t r0 = 0; r0 < run.rows && ce == cudaSuccess; r0 += range) {
            const size_t rows_now = std::min(range, run.rows - r0);
            size_t tables = predictions;
            for (size_t v = 0; v < views.size(); ++v) {
                const DeviceBatch& db = views[v].batch;
                EvalProblem prob = make_problem(plan, run, 0);
                prob.fast_math = r->fast_math;
                prob.input += r0;
                prob.num_rows = rows_now;
                /* SbProgram::index is the program's position in the run: shift the base so that the batch's first program lands on row 0 */
                prob.output = reinterpret_cast<float*>(reinterpret_cast<uintptr_t>(scratch) - first_program * range * sizeof(float));
                prob.out_program_stride = range;
                LaunchPlan lp = plan_launch(db, prob, r->sm_count, r->smem_limit, r->scratch_limit);
                if (!lp.ok) {
                    r->last_error = "program batch does not fit shared memory";
                    return lp.overflow ? SECANT_ERROR_OVERFLOW : SECANT_ERROR_REGISTER_OVERFLOW;
                }
                if (tables_made[v] == lp.variant) lp.table_elements = 0;
                tables_made[v] = lp.variant;
                unsigned launches = 0;
                ce = launch_eval(db, prob, lp, scratch + tables, stream, &launches);
                tables += 4 * db.total_cst;
                g_kernel_launches.fetch_add(launches);
                if (ce != cudaSuccess) break;
            }
            if (ce == cudaSuccess)
                ce = launch_gram(scratch, range, (uint32_t)rows_now, reinterpret_cast<const float*>(run.targets.address) + r0,
                                 run.targets.leading_dimension, (uint32_t)run.num_targets, (uint32_t)cohort, (uint32_t)batch_programs,
                                 reinterpret_cast<float*>(run.output.address) + (first_program / cohort) * run.output.leading_dimension,
                                 run.output.leading_dimension, stream);
        }
        if (ce == cudaSuccess && done) ce = cudaEventRecord((*done)[k], stream);
        if (ce != cudaSuccess) return cuda_fail(r, ce, "kernel launch");
        if (used) (*used)[k] = 1;
    }
    return SECANT_SUCCESS;
}

/* Waits for everything the runner has enqueued; false (and a destroy-only handle) when a wait fails. */
bool drain_streams(SecantCubinRunnerImpl* r) {
    bool ok = true;
    for (auto& s : r->streams) ok = (cudaStreamSynchronize(s) == cudaSuccess) && ok;
    ok = (cudaStreamSynchronize(r->copy_stream) == cudaSuccess) && ok;
    if (!ok) r->failed = true;
    return ok;
}

/* Waits until every compute stream that touched the slot has finished with it. */
SecantResult retire_slot(SecantCubinRunnerImpl* r, Slot& s, bool* unknown) {
    SecantResult result = SECANT_SUCCESS;
    for (size_t k = 0; k < s.done.size(); ++k) {
        if (!s.used[k]) continue;
        const cudaError_t e = cudaEventSynchronize(s.done[k]);
        if (e != cudaSuccess) { result = cuda_fail(r, e, "waiting for a batch"); *unknown = true; }
        s.used[k] = 0;
    }
    return result;
}

/* Zeroes the output vectors of the programs from `first` on.  The evaluator writes every active bin of
 * a program it was launched for, so only a call that fails half way has something to clear: the
 * reference clears every vector before it starts (projects/secant/s_cubin_runner.c:243-286). */
SecantResult clear_outputs(SecantCubinRunnerImpl* r, const std::vector<UnpackedRun>& runs, size_t first) {
    for (const auto& run : runs) {
        const size_t vectors = run.output_count / run.programs.asts.count; /* per program (targets) */
        const size_t at = first * vectors;
        if (at >= run.output_count) continue;
        SB_CUDA(cudaMemset2DAsync(reinterpret_cast<float*>(run.output.address) + at * run.output.leading_dimension,
                                  run.output.leading_dimension * sizeof(float), 0, run.output_width * sizeof(float),
                                  run.output_count - at, r->streams[0]),
                "clearing output");
    }
    return SECANT_SUCCESS;
}

/* Joins the compute streams that were used into stream 0, waits for it and reads the device time. */
cudaError_t finish_streams(SecantCubinRunnerImpl* r, size_t streams_used, double* seconds) {
    cudaError_t ce = cudaSuccess;
    for (size_t k = 1; k < std::min(streams_used, r->streams.size()) && ce == cudaSuccess; ++k) {
        ce = cudaEventRecord(r->ev_join, r->streams[k]);
        if (ce == cudaSuccess) ce = cudaStreamWaitEvent(r->streams[0], r->ev_join, 0);
    }
    if (ce == cudaSuccess) ce = cudaEventRecord(r->ev_stop, r->streams[0]);
    if (ce == cudaSuccess) ce = cudaEventSynchronize(r->ev_stop);
    float ms = 0;
    if (ce == cudaSuccess) ce = cudaEventElapsedTime(&ms, r->ev_start, r->ev_stop);
    *seconds = ms * 1e-3;
    return ce;
}

SecantResult execute(SecantCubinRunnerImpl* r, const std::vector<UnpackedRun>& runs, const ProgramRules& rules,
                     SecantRunnerStats* stats) {
    const SecantCubinPlan& plan = *r->plan;
    const SecantAstProgramSet& programs = runs[0].programs;
    const size_t P = programs.asts.count;
    uint8_t arity[SECANT_AST_MAX_ROUTINES];
    SecantResult result = routine_arities(programs.routines, arity);
    if (result != SECANT_SUCCESS) {
        const SecantResult scan = P <= kMinBatch ? preflight_all(programs.asts, rules) : SECANT_SUCCESS;
        return scan != SECANT_SUCCESS ? scan : result;
    }
    if ((uint64_t)P > 0xffffffffull) return SECANT_ERROR_OVERFLOW;

    const double t_begin = now_seconds();
    size_t batch_size = (P + 3) / 4;
    if (batch_size < kMinBatch) batch_size = kMinBatch;
    const bool gram = plan.shape == SECANT_KERNEL_SHAPE_STATIC_GRAM_STATS_F32;
    if (gram) batch_size = (batch_size + plan.asts_per_kernel - 1) / plan.asts_per_kernel * plan.asts_per_kernel; /* whole cohorts */
    if (batch_size > P) batch_size = P;
    const size_t num_batches = (P + batch_size - 1) / batch_size;
    const bool accumulate = plan.shape != SECANT_KERNEL_SHAPE_STATIC_MATERIALIZE_F32;

    const size_t threads = r->workers.size() + 1;
    const size_t piece_size = std::min(kPieceMax, std::max(kPieceMin, batch_size / (threads * kPiecesPerThread)));
    const size_t pieces_per_batch = (batch_size + piece_size - 1) / piece_size;
    auto pieces_of = [&](size_t batch) { return (std::min(batch_size, P - batch * batch_size) + piece_size - 1) / piece_size; };
    auto open_slot = [&](Slot& s, size_t batch) { /* under the mutex; grows the piece list only while no job runs on it */
        prepare_slot(s, std::min(batch_size, P - batch * batch_size));
        s.used_pieces = pieces_of(batch);
        s.done_pieces = 0;
    };

    SB_CUDA(cudaEventRecord(r->ev_start, r->streams[0]), "cudaEventRecord");
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        for (size_t k = 0; k < r->slots.size(); ++k) {
            Slot& s = r->slots[k];
            std::fill(s.used.begin(), s.used.end(), 0);
            if (k >= num_batches) continue;
            if (s.pieces.size() < pieces_per_batch) s.pieces.resize(pieces_per_batch);
            open_slot(s, k);
        }
        std::fill(r->worker_seconds.begin(), r->worker_seconds.end(), 0.0);
        r->job_programs = &programs;
        r->job_arity = arity;
        r->job_rules = rules;
        r->job_batch_size = batch_size;
        r->job_piece_size = piece_size;
        r->job_pieces_per_batch = pieces_per_batch;
        r->job_num_pieces = (num_batches - 1) * pieces_per_batch + pieces_of(num_batches - 1);
        r->job_next_piece = 0;
        r->job_open_batches = std::min(num_batches, r->slots.size());
        r->job_encode_seconds = 0;
        r->job_abort = false;
        r->job_active = true;
    }
    if (P > piece_size) r->cv_work.notify_all(); /* a single piece is the calling thread's own */
    /* Whatever way this function is left (a result code or an exception from a container), the
     * workers must be off this job first: they read `arity`, `programs` and `rules`, which live in
     * the caller's frames. */
    struct JobGuard {
        SecantCubinRunnerImpl* r;
        ~JobGuard() {
            std::unique_lock<std::mutex> lock(r->mutex);
            end(lock);
        }
        void end(std::unique_lock<std::mutex>& lock) {
            r->job_abort = true;
            r->cv_ready.wait(lock, [&] { return r->job_encoding == 0; });
            r->job_active = false;
        }
    } job_guard{r};

    bool unknown = false;
    size_t launched_batches = 0, retired_batches = 0, stream_cursor = 0;
    double upload_seconds = 0, wait_seconds = 0, encode_sum = 0;
    std::vector<View> views;
    const auto retire = [&]() { /* the oldest batch in flight: wait for it and open its slot for the batch that comes next to it */
        Slot& old = r->slots[retired_batches % r->slots.size()];
        const double t_wait = now_seconds();
        const SecantResult w = retire_slot(r, old, &unknown);
        wait_seconds += now_seconds() - t_wait;
        if (result == SECANT_SUCCESS) result = w;
        const size_t next = retired_batches++ + r->slots.size();
        if (next >= num_batches) return;
        {
            std::lock_guard<std::mutex> lock(r->mutex);
            open_slot(old, next);
            r->job_open_batches = next + 1;
        }
        r->cv_work.notify_all();
    };
    for (size_t b = 0; b < num_batches && result == SECANT_SUCCESS; ++b) {
        Slot& slot = r->slots[b % r->slots.size()];
        {
            std::unique_lock<std::mutex> lock(r->mutex);
            while (slot.done_pieces < slot.used_pieces) {
                const size_t piece = take_piece(r); /* nothing to launch yet: help */
                if (piece != SIZE_MAX) encode_piece(r, lock, piece, &r->worker_seconds.back());
                else r->cv_ready.wait(lock);
            }
            for (size_t q = 0; q < slot.used_pieces && result == SECANT_SUCCESS; ++q) result = slot.pieces[q].status; /* the first in program order */
        }
        if (result != SECANT_SUCCESS) {
            const SecantResult scan = P <= kMinBatch ? preflight_all(programs.asts, rules) : SECANT_SUCCESS;
            if (scan != SECANT_SUCCESS) return scan; /* nothing has been touched (a gram run's statistics are cleared after this point) */
            break;
        }
        const double t_up = now_seconds();
        result = upload_batch(r, slot, &views);
        upload_seconds += now_seconds() - t_up;
        if (result != SECANT_SUCCESS) break;
        std::vector<cudaEvent_t>* done = num_batches > 2 ? &slot.done : nullptr; /* only a batch whose slot is used again is waited for by itself */
        if (gram && b == 0) { /* its statistics are added to range by range: the active entries start from zero */
            result = clear_outputs(r, runs, 0);
            cudaError_t ce = result == SECANT_SUCCESS ? cudaEventRecord(r->ev_join, r->streams[0]) : cudaSuccess;
            for (size_t k = 1; k < r->streams.size() && ce == cudaSuccess; ++k) ce = cudaStreamWaitEvent(r->streams[k], r->ev_join, 0);
            if (ce != cudaSuccess) result = cuda_fail(r, ce, "clearing statistics");
            if (result != SECANT_SUCCESS) break;
        }
        if (gram) {
            const size_t first = b * batch_size;
            result = launch_gram_batch(r, views, runs, first, std::min(batch_size, P - first), &stream_cursor, slot.uploaded, done, &slot.used);
        } else {
            result = launch_batch(r, views, static_cast<const SbProgram*>(slot.pinned), runs, &stream_cursor, slot.uploaded, done, &slot.used);
        }
        if (result != SECANT_SUCCESS) break;
        ++launched_batches;
        /* recycle the oldest batch once two are queued behind it, so there is always a slot to encode into */
        while (launched_batches - retired_batches > 2 && result == SECANT_SUCCESS) retire();
    }
    /* stop the workers' job, then drain what is still running */
    {
        std::unique_lock<std::mutex> lock(r->mutex);
        job_guard.end(lock);
        encode_sum = r->job_encode_seconds;
    }
    const double t_wait = now_seconds();
    if (result != SECANT_SUCCESS && !unknown) { /* nothing of the call stays in flight, and what was not scored reads zero */
        if (!drain_streams(r)) unknown = true;
        else if (accumulate) (void)clear_outputs(r, runs, launched_batches * batch_size);
    }
    if (!unknown) {
        const cudaError_t ce = finish_streams(r, result == SECANT_SUCCESS ? stream_cursor : r->streams.size(), &stats->runtime_seconds);
        if (ce != cudaSuccess) { const SecantResult w = cuda_fail(r, ce, "completion"); unknown = true; if (result == SECANT_SUCCESS) result = w; }
    }
    wait_seconds += now_seconds() - t_wait;
    stats->compile_critical_seconds = *std::max_element(r->worker_seconds.begin(), r->worker_seconds.end());
    /* module counts in the reference's unit, a recipe-capacity worth of programs (callers such as
     * projects/secant/tests/toggle_cuda_test.c:245 check them); batches here are much larger */
    {
        const size_t capacity = std::max<size_t>(1, r->plan->num_kernels * r->plan->asts_per_kernel);
        const size_t launched_programs = std::min<size_t>(P, launched_batches * batch_size);
        stats->num_modules = (P + capacity - 1) / capacity;
        stats->modules_loaded = (launched_programs + capacity - 1) / capacity;
    }
    stats->num_asts = P;
    stats->compile_work_seconds = encode_sum;
    stats->compile_window_seconds = now_seconds() - t_begin - wait_seconds;
    stats->module_load_seconds = upload_seconds;
    stats->completion_wait_seconds = wait_seconds;
    stats->module_unload_seconds = 0;
    if (unknown) {
        r->failed = true;
        return SECANT_ERROR_COMPLETION_UNKNOWN;
    }
    return result;
}

}  // namespace

extern "C" {

SecantResult secant_cubin_runner_create(const SecantCubinPlan* plan, const void* cubin, size_t cubin_size,
                                        const SecantCubinRunnerOptions* options, SecantCubinRunner* runner_ret) {
    if (!runner_ret) return SECANT_ERROR_INVALID_VALUE;
    *runner_ret = nullptr;
    if (!plan || plan->magic != kPlanMagic || !cubin || cubin_size != plan->cubin_size || !options ||
        options->struct_size < sizeof(*options))
        return SECANT_ERROR_INVALID_VALUE;
    const SecantResult o = options_validate(options);
    if (o != SECANT_SUCCESS) return o;
    SecantCubinRunnerImpl* r = SB_FAULT("alloc") ? nullptr : new (std::nothrow) SecantCubinRunnerImpl();
    if (!r) return SECANT_ERROR_ALLOCATION_FAILED;
    r->plan = plan;
    return create_common(r, options, runner_ret);
}

SecantResult secant_b200_runner_create(const SecantCubinRecipeHeader* recipe, const SecantCubinRunnerOptions* options,
                                       SecantCubinRunner* runner_ret) {
    if (!runner_ret) return SECANT_ERROR_INVALID_VALUE;
    *runner_ret = nullptr;
    const SecantResult v = recipe_validate(recipe);
    if (v != SECANT_SUCCESS) return v;
    const SecantResult o = options_validate(options);
    if (o != SECANT_SUCCESS) return o;
    SecantCubinRunnerImpl* r = SB_FAULT("alloc") ? nullptr : new (std::nothrow) SecantCubinRunnerImpl();
    if (!r) return SECANT_ERROR_ALLOCATION_FAILED;
    plan_fill(&r->owned_plan, recipe, 0);
    r->plan = &r->owned_plan;
    return create_common(r, options, runner_ret);
}

SecantResult secant_cubin_runner_run_batch(SecantCubinRunner r, const SecantCubinRunHeader* const* headers, size_t count,
                                           SecantRunnerStats* stats) {
    SecantRunnerStats measured = secant_runner_stats_init();
    const double begin = now_seconds();
    if (stats) {
        if (stats->struct_size < sizeof(*stats) || stats->flags || stats->reserved) return SECANT_ERROR_INVALID_VALUE;
        if (stats->version != SECANT_RUNNER_STATS_VERSION_1) return SECANT_ERROR_UNSUPPORTED_VERSION;
        measured.struct_size = stats->struct_size;
        std::memcpy(stats, &measured, sizeof(measured)); /* zero counters, trailing bytes untouched */
    }
    if (!r || !headers || !count || count > SIZE_MAX / sizeof(UnpackedRun)) return SECANT_ERROR_INVALID_VALUE;
    bool ok = false;
    void* ctx = current_context(&ok);
    if (!ok || ctx != r->context) return SECANT_ERROR_INVALID_STATE;
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        if (r->active || r->failed || r->shutdown) return SECANT_ERROR_INVALID_STATE;
        r->active = true;
    }
    SecantResult result = SECANT_SUCCESS;
    std::vector<UnpackedRun> runs;
    try {
        if (SB_FAULT("alloc")) throw std::bad_alloc();
        runs.resize(count);
    } catch (...) {
        result = SECANT_ERROR_ALLOCATION_FAILED;
    }
    for (size_t i = 0; result == SECANT_SUCCESS && i < count; ++i) result = run_unpack(*r->plan, headers[i], &runs[i]);
    ProgramRules rules;
    /* a run of one batch is encoded before anything is touched, and the encoder makes the scan's checks on
     * the way: execute() scans only when the encoder found something (0.45 ms of 2.5 for 3,000 programs) */
    if (result == SECANT_SUCCESS)
        result = runs_validate(*r->plan, runs.data(), count, &rules, runs[0].programs.asts.count <= kMinBatch ? SCAN_ROUTINES : SCAN_EVERYTHING);
    if (result == SECANT_SUCCESS) {
        try {
            result = execute(r, runs, rules, &measured);
        } catch (const std::bad_alloc&) {
            /* work already enqueued still reads the caller's buffers: wait for it before handing them back */
            result = drain_streams(r) ? SECANT_ERROR_ALLOCATION_FAILED : SECANT_ERROR_COMPLETION_UNKNOWN;
        }
    }
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        r->active = false;
    }
    if (measured.num_modules) measured.total_seconds = now_seconds() - begin;
    if (stats) std::memcpy(stats, &measured, sizeof(measured));
    return result;
}

SecantResult secant_cubin_runner_run(SecantCubinRunner r, const SecantCubinRunHeader* run, SecantRunnerStats* stats) {
    return secant_cubin_runner_run_batch(r, &run, 1, stats);
}

SecantResult secant_cubin_runner_destroy(SecantCubinRunner r) {
    if (!r) return SECANT_SUCCESS;
    bool ok = false;
    void* ctx = current_context(&ok);
    if (r->context && (!ok || ctx != r->context)) return SECANT_ERROR_INVALID_STATE;
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        if (r->active || r->populations) return SECANT_ERROR_INVALID_STATE; /* populations hold a pointer to their runner */
    }
    const SecantResult result = runner_teardown(r);
    if (result != SECANT_SUCCESS) { r->failed = true; return result; }
    delete r;
    return SECANT_SUCCESS;
}

const char* secant_b200_runner_last_error(SecantCubinRunner r) { return r ? r->last_error.c_str() : ""; }

uint64_t secant_b200_kernel_launch_count(void) { return g_kernel_launches.load(); }
uint64_t secant_b200_row_stream_bytes(void) { return g_row_stream_bytes.load(); }

}  // extern "C"

/* ---- device-resident populations ------------------------------------------------------ */

namespace {

size_t program_length(const SecantAstInstruction* code) {
    size_t at = 0;
    for (size_t n = 0; n < SECANT_AST_MAX_PROGRAM_INSTRUCTIONS; ++n) {
        const size_t width = secant_ast_instruction_size_get(code + at);
        if (!width) return 0;
        const bool last = code[at] == SECANT_AST_INSTRUCTION_TYPE_RETURN_F32;
        at += width;
        if (last) return at;
    }
    return 0;
}

SecantResult copy_programs(const SecantAstProgramList& list, std::vector<uint8_t>* bytes, std::vector<const uint8_t*>* ptrs) {
    std::vector<size_t> offsets(list.count);
    for (size_t i = 0; i < list.count; ++i) {
        if (!list.items[i]) return SECANT_ERROR_BAD_PROGRAM;
        const size_t n = program_length(list.items[i]);
        if (!n) return SECANT_ERROR_BAD_PROGRAM;
        offsets[i] = bytes->size();
        bytes->insert(bytes->end(), list.items[i], list.items[i] + n);
    }
    ptrs->resize(list.count);
    for (size_t i = 0; i < list.count; ++i) (*ptrs)[i] = bytes->data() + offsets[i];
    return SECANT_SUCCESS;
}

SecantResult execute_resident(SecantCubinRunnerImpl* r, SecantB200PopulationImpl* pop, const std::vector<UnpackedRun>& runs,
                              SecantRunnerStats* stats) {
    const SecantCubinPlan& plan = *r->plan;
    SB_CUDA(cudaEventRecord(r->ev_start, r->streams[0]), "cudaEventRecord");
    size_t cursor = 0;
    SecantResult result = SECANT_SUCCESS;
    for (auto& b : pop->batches) {
        result = launch_batch(r, b.views, b.headers.data(), runs, &cursor, nullptr, nullptr, nullptr);
        if (result != SECANT_SUCCESS) break;
    }
    if (result != SECANT_SUCCESS && plan.shape != SECANT_KERNEL_SHAPE_STATIC_MATERIALIZE_F32 && drain_streams(r)) (void)clear_outputs(r, runs, 0);
    const double t_wait = now_seconds();
    const cudaError_t ce = finish_streams(r, result == SECANT_SUCCESS ? cursor : r->streams.size(), &stats->runtime_seconds);
    stats->completion_wait_seconds = now_seconds() - t_wait;
    {
        const size_t capacity = std::max<size_t>(1, r->plan->num_kernels * r->plan->asts_per_kernel);
        stats->num_modules = stats->modules_loaded = (pop->set.asts.count + capacity - 1) / capacity;
    }
    stats->num_asts = pop->set.asts.count;
    if (ce != cudaSuccess) {
        cuda_fail(r, ce, "completion");
        r->failed = true;
        return SECANT_ERROR_COMPLETION_UNKNOWN;
    }
    return result;
}

}  // namespace

extern "C" {

SecantResult secant_b200_population_create(SecantCubinRunner r, const SecantAstProgramSet* programs, uint32_t toggle_bits,
                                           SecantB200Population* population_ret) {
    if (!population_ret) return SECANT_ERROR_INVALID_VALUE;
    *population_ret = nullptr;
    if (!r || !programs || !programs->asts.count || !programs->asts.items || toggle_bits > 32u ||
        programs->routines.count > SECANT_AST_MAX_ROUTINES || (programs->routines.count && !programs->routines.items) ||
        (uint64_t)programs->asts.count > 0xffffffffull)
        return SECANT_ERROR_INVALID_VALUE;
    bool ok = false;
    void* ctx = current_context(&ok);
    if (!ok || ctx != r->context) return SECANT_ERROR_INVALID_STATE;
    const SecantCubinPlan& plan = *r->plan;
    if (plan.shape == SECANT_KERNEL_SHAPE_STATIC_GRAM_STATS_F32) return SECANT_ERROR_UNSUPPORTED_SHAPE; /* cohorts go through the run entry points */
    ProgramRules rules;
    rules.num_columns = plan.num_inputs;
    rules.num_constants = plan.num_constants;
    rules.banks_allowed = plan.shape == SECANT_KERNEL_SHAPE_TOGGLE_SSE_F32;
    rules.toggle_bits = rules.banks_allowed ? toggle_bits : 0;
    rules.split_parts = true;
    rules.hoist_bank = true;
    rules.number_bits = true;
    rules.hoist_row = rules.banks_allowed; /* a population is usually scored against many banks */
    for (size_t i = 0; i < programs->routines.count; ++i) {
        const SecantResult s = preflight(programs->routines.items[i], rules);
        if (s != SECANT_SUCCESS) return s;
    }
    for (size_t i = 0; i < programs->asts.count; ++i) {
        const SecantResult s = preflight(programs->asts.items[i], rules);
        if (s != SECANT_SUCCESS) return s;
    }
    uint8_t arity[SECANT_AST_MAX_ROUTINES];
    SecantResult result = routine_arities(programs->routines, arity);
    if (result != SECANT_SUCCESS) return result;
    SecantB200PopulationImpl* pop = new (std::nothrow) SecantB200PopulationImpl();
    if (!pop) return SECANT_ERROR_ALLOCATION_FAILED;
    pop->runner = r;
    pop->toggle_bits = toggle_bits;
    Slot staging; /* reuses the upload helper; its device buffers are handed to the population */
    try {
        result = copy_programs(programs->routines, &pop->routine_bytes, &pop->routine_ptrs);
        if (result == SECANT_SUCCESS) result = copy_programs(programs->asts, &pop->ast_bytes, &pop->ast_ptrs);
        pop->set.routines.items = pop->routine_ptrs.data();
        pop->set.routines.count = pop->routine_ptrs.size();
        pop->set.asts.items = pop->ast_ptrs.data();
        pop->set.asts.count = pop->ast_ptrs.size();
        const size_t P = programs->asts.count;
        size_t batch_size = (P + 3) / 4;
        if (batch_size < kMinBatch) batch_size = kMinBatch;
        if (batch_size > P) batch_size = P;
        staging.pieces.resize(1);
        staging.used_pieces = 1;
        for (size_t first = 0; first < P && result == SECANT_SUCCESS; first += batch_size) {
            const size_t count = std::min(batch_size, P - first);
            EncodedBatch& enc = staging.pieces[0].enc;
            enc.clear();
            for (size_t i = 0; i < count && result == SECANT_SUCCESS; ++i) {
                result = encode_program(programs->asts.items[first + i], programs->routines, arity, rules, enc);
                if (result == SECANT_SUCCESS) enc.programs.back().index = (uint32_t)(first + i);
            }
            if (result != SECANT_SUCCESS) break;
            for (const auto& p : enc.programs) pop->total_ops += p.n_ops;
            if (!staging.uploaded && cudaEventCreateWithFlags(&staging.uploaded, cudaEventDisableTiming) != cudaSuccess) {
                result = SECANT_ERROR_DRIVER_FAILED;
                break;
            }
            SecantB200PopulationImpl::Resident res;
            prepare_slot(staging, count);
            staging.packing = false; /* encoded as one piece, before there are buffers */
            result = upload_batch(r, staging, &res.views);
            if (result != SECANT_SUCCESS) break;
            if (cudaStreamSynchronize(r->copy_stream) != cudaSuccess) { result = SECANT_ERROR_DRIVER_FAILED; break; }
            res.headers.assign(static_cast<const SbProgram*>(staging.pinned), static_cast<const SbProgram*>(staging.pinned) + count);
            pop->batches.reserve(pop->batches.size() + 1);
            res.device = staging.device; /* keep this allocation; the next batch gets a new one */
            staging.device = nullptr;
            staging.device_cap = 0;
            pop->batches.push_back(std::move(res));
        }
    } catch (const std::bad_alloc&) {
        result = SECANT_ERROR_ALLOCATION_FAILED;
    }
    if (staging.pinned) cudaFreeHost(staging.pinned);
    if (staging.device) cudaFree(staging.device);
    if (staging.uploaded) cudaEventDestroy(staging.uploaded);
    if (result != SECANT_SUCCESS) {
        for (auto& b : pop->batches) cudaFree(b.device);
        delete pop;
        return result;
    }
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        ++r->populations;
    }
    *population_ret = pop;
    return SECANT_SUCCESS;
}

SecantResult secant_b200_population_run_batch(SecantB200Population pop, const SecantCubinRunHeader* const* headers, size_t count,
                                              SecantRunnerStats* stats) {
    SecantRunnerStats measured = secant_runner_stats_init();
    const double begin = now_seconds();
    if (stats) {
        if (stats->struct_size < sizeof(*stats) || stats->flags || stats->reserved) return SECANT_ERROR_INVALID_VALUE;
        if (stats->version != SECANT_RUNNER_STATS_VERSION_1) return SECANT_ERROR_UNSUPPORTED_VERSION;
        measured.struct_size = stats->struct_size;
        std::memcpy(stats, &measured, sizeof(measured));
    }
    if (!pop || !headers || !count) return SECANT_ERROR_INVALID_VALUE;
    SecantCubinRunnerImpl* r = pop->runner;
    bool ok = false;
    void* ctx = current_context(&ok);
    if (!ok || ctx != r->context) return SECANT_ERROR_INVALID_STATE;
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        if (r->active || r->failed || r->shutdown) return SECANT_ERROR_INVALID_STATE;
        r->active = true;
    }
    SecantResult result = SECANT_SUCCESS;
    std::vector<UnpackedRun> runs;
    try {
        runs.resize(count);
    } catch (...) {
        std::lock_guard<std::mutex> lock(r->mutex);
        r->active = false;
        return SECANT_ERROR_ALLOCATION_FAILED;
    }
    bool same_bits = true;
    for (size_t i = 0; result == SECANT_SUCCESS && i < count; ++i) {
        /* the request's program views are replaced by the population's own */
        alignas(16) unsigned char copy[sizeof(SecantB200ToggleSSERun) + 64];
        const SecantCubinRunHeader* h = headers[i];
        if (!h || h->struct_size < sizeof(*h) + sizeof(SecantAstProgramSet)) { result = SECANT_ERROR_INVALID_VALUE; break; }
        const size_t n = std::min<size_t>(h->struct_size, sizeof(copy));
        std::memcpy(copy, h, n);
        reinterpret_cast<SecantCubinRunHeader*>(copy)->struct_size = (uint32_t)n;
        std::memcpy(copy + sizeof(SecantCubinRunHeader), &pop->set, sizeof(pop->set));
        result = run_unpack(*r->plan, reinterpret_cast<const SecantCubinRunHeader*>(copy), &runs[i]);
        same_bits = same_bits && runs[i].toggle_bits == pop->toggle_bits;
    }
    ProgramRules rules;
    if (result == SECANT_SUCCESS) result = runs_validate(*r->plan, runs.data(), count, &rules, same_bits ? SCAN_NOTHING : SCAN_EVERYTHING);
    if (result == SECANT_SUCCESS && !same_bits && rules.toggle_bits < pop->toggle_bits) {
        /* records were encoded for pop->toggle_bits; fewer bits would leave stale patch sites unchecked */
        result = SECANT_ERROR_BAD_PROGRAM;
    }
    if (result == SECANT_SUCCESS) {
        try {
            result = execute_resident(r, pop, runs, &measured);
        } catch (const std::bad_alloc&) {
            result = drain_streams(r) ? SECANT_ERROR_ALLOCATION_FAILED : SECANT_ERROR_COMPLETION_UNKNOWN;
        }
    }
    {
        std::lock_guard<std::mutex> lock(r->mutex);
        r->active = false;
    }
    if (measured.num_modules) measured.total_seconds = now_seconds() - begin;
    if (stats) std::memcpy(stats, &measured, sizeof(measured));
    return result;
}

SecantResult secant_b200_population_run(SecantB200Population pop, const SecantCubinRunHeader* run, SecantRunnerStats* stats) {
    return secant_b200_population_run_batch(pop, &run, 1, stats);
}

uint64_t secant_b200_population_num_ops(SecantB200Population pop) { return pop ? pop->total_ops : 0; }

SecantResult secant_b200_population_destroy(SecantB200Population pop) {
    if (!pop) return SECANT_SUCCESS;
    SecantResult result = SECANT_SUCCESS;
    for (auto& b : pop->batches)
        if (b.device && cudaFree(b.device) != cudaSuccess) result = SECANT_ERROR_DRIVER_FAILED;
    {
        std::lock_guard<std::mutex> lock(pop->runner->mutex);
        if (pop->runner->populations) --pop->runner->populations;
    }
    delete pop;
    return result;
}

SecantResult secant_b200_runner_set_math(SecantCubinRunner r, uint32_t mode) {
    if (!r || mode > SECANT_B200_MATH_FAST) return SECANT_ERROR_INVALID_VALUE;
    std::lock_guard<std::mutex> lock(r->mutex);
    if (r->active) return SECANT_ERROR_INVALID_STATE;
    r->fast_math = mode == SECANT_B200_MATH_FAST ? 1u : 0u;
    return SECANT_SUCCESS;
}

SecantResult secant_b200_runner_set_scratch_limit(SecantCubinRunner r, size_t bytes) {
    if (!r) return SECANT_ERROR_INVALID_VALUE;
    std::lock_guard<std::mutex> lock(r->mutex);
    if (r->active) return SECANT_ERROR_INVALID_STATE;
    r->scratch_limit = bytes ? std::max<size_t>(1, bytes / sizeof(float)) : kDefaultScratchFloats;
    return SECANT_SUCCESS;
}

}  // extern "C"
