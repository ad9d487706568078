/*
 * planner.cpp - launch geometry of the population evaluator: register-tile variant, warps per
 * CTA, staged tile size, programs per CTA, row splits, and the shared-memory layout that follows.
 * Host-only arithmetic, so the CPU test-suite can check its bounds without a device.
 *
 * The reference sizes its launches from the recipe (projects/secant/s_runner_pipeline.c:259-283:
 * grid = row tiles x configuration blocks).  Here a CTA owns a set of programs and a range of
 * rows; it walks the range tile by tile and its warps take (program, permutation) items from a
 * queue for every tile.
 */
#include "evaluator.cuh"

#include <algorithm>
#include <cmath>

namespace sb {

namespace {

uint32_t round16(size_t v) { return (uint32_t)((v + 15) / 16 * 16); }

uint32_t quantities(const EvalProblem& prob) {
    return prob.mode == EVAL_AFFINE_STATS ? prob.num_targets + 2u : prob.num_targets;
}

}  // namespace

Geom make_geom(const DeviceBatch& batch, const EvalProblem& prob, const LaunchPlan& plan) {
    const uint32_t rr = (uint32_t)kVariantRows[plan.variant], rc = (uint32_t)kVariantBanks[plan.variant];
    const uint32_t ncols = prob.num_inputs + (prob.mode == EVAL_MATERIALIZE ? 0u : prob.num_targets);
    const uint32_t gpi = plan.groups_per_item ? plan.groups_per_item : 1u;
    const uint32_t ppi = plan.perms_per_item ? plan.perms_per_item : 1u;
    const uint32_t slots = batch.max_slots + (batch.uses_scratch ? 1u : 0u);
    Geom g;
    g.tile_rows = plan.tile_rows;
    g.tile_buffers = plan.tile_buffers;
    g.tile_bytes = round16((size_t)ncols * plan.tile_rows * 4);
    g.num_groups = plan.num_groups;
    g.row_splits = plan.row_splits;
    g.groups_per_item = gpi;
    g.perms_per_item = ppi;
    g.parts = plan.parts ? plan.parts : 1u;
    g.passes_per_part = (plan.tile_rows / (32u * rr) + g.parts - 1) / g.parts;
    g.exec_bytes = round16(((size_t)batch.max_insn + 1) * sizeof(SbInsn));
    g.table_bytes = round16((size_t)std::max<uint32_t>(1u, ppi * gpi * batch.max_cst * rc) * 4);
    g.hoist_bytes = round16((size_t)batch.max_hoisted * 32u * rr * 4);
    g.slot_bytes = round16((size_t)slots * rr * rc * 128u);
    g.psum_bytes = round16((size_t)std::max<uint32_t>(1u, quantities(prob) * ppi * gpi * rc) * 4);
    g.warp_bytes = g.exec_bytes + g.table_bytes + g.hoist_bytes + g.slot_bytes + g.psum_bytes;
    g.scratch_slot = batch.max_slots; /* one slot beyond what the programs use */
    g.rows_per_split = plan.rows_per_split;
    g.direct = 0;
    return g;
}

namespace {

size_t smem_needed(const Geom& g, uint32_t warps) { return (size_t)g.tile_bytes * g.tile_buffers + 16 + (size_t)g.warp_bytes * warps; }

/* How a launch is cut into tiles, CTAs and queue items when it is small.
 *
 * The rules above it aim at large launches, whose grid is many waves deep.  With few programs or rows they gave
 * grids of 150 CTAs on 148 SMs (two waves for one), a dozen items for twenty warps, half the warps because a
 * second tile buffer was reserved that a CTA of one tile does not use, or a CTA with two items on every SM of the
 * machine.  Here the cut with the shortest estimated time is taken: the grid's waves times a CTA's rounds of items.
 * The constants are issue slots, measured on the 64-set population: 330 for one pass of the main part with
 * its loss, about 900 to set an item up, and a warp that issues every seventh cycle when alone; an SM
 * issues 2.6 per cycle at best.  (A launch whose programs read few of the run's toggle bits is small in this sense
 * too.)  The order in which rows are added does not follow the cut: where its rows are not the rules', the launch keeps the
 * total of every pass, which is the same number in any cut, and they are added as the rules' tiles and splits would add them
 * (combine_passes_kernel in evaluator.cu).  With toggles, whose kernel keeps no such totals, and where there is no room for
 * them, the rows stay the rules'.
 * Tiles of half the rows, CTAs of several tiles and parts of tiles are tried since a CTA of 19 items on 20 warps ends
 * with its longest program: 124 programs x 8 sets x 47,735 rows 320 -> 197 us a call, 488 x 16 x 5,823 191 -> 145, 124 x
 * 3 x 19,735 163 -> 155 (all with their few heavy programs in the same launch, see views_to_launch in runner.cpp). */
struct Cut {
    uint32_t tile_rows, tiles_per_split, splits, warps; /* tiles_per_split: tiles a CTA walks */
    uint32_t gpi, ppi, parts; /* parts only without toggles: the permutations are cuts enough, and their kernel has no room for it */
    unsigned long long groups;
};
struct Work { unsigned long long programs, bank_groups; double perms, most_perms; uint32_t passes; double prelude; /* issue slots of a pass */ int sms; double longest; /* the costliest program over the average */ }; /* perms: of a program, on the average and at most */

double cut_cycles(const Cut& cut, const Work& w) {
    const double per_cta = (double)((w.programs + cut.groups - 1) / cut.groups);
    const double chunks = (double)(w.bank_groups / cut.gpi * cut.parts); /* items of a permutation, or of cut.ppi of them */
    const double each = chunks * std::max(1.0, w.perms / cut.ppi), largest = chunks * std::max(1.0, w.most_perms / cut.ppi);
    const double items = std::ceil((per_cta - 1.0) * each + largest), empty = std::max(0.0, per_cta * largest - items);
    const double active = std::min<double>(cut.warps, items);
    const double rate = std::min(0.14, 2.6 / active);
    const uint32_t passes = (w.passes + cut.parts - 1) / cut.parts;
    const auto slots = [&](double n, double groups) { return 900.0 * n + passes * (w.prelude * n + 330.0 * groups); };
    const double item = slots(1.0, cut.gpi * std::min<double>(cut.ppi, w.most_perms));
    const unsigned long long grid = cut.groups * cut.splits;
    const auto cta = [&](double time) { return 3000.0 + cut.tiles_per_split * (1500.0 + time / rate + empty * 400.0 / cut.warps); };
    if (w.perms < w.most_perms) { /* uneven: an average CTA for the work, the one with most permutations for the end */
        const auto time = [&](double n, double all_perms) { return std::max(item, slots(n, chunks * cut.gpi * all_perms) / cut.warps + 0.5 * item); };
        const double last = cta(time(items, (per_cta - 1.0) * w.perms + w.most_perms));
        return std::max(last, cta(time(std::ceil(per_cta * each), per_cta * w.perms)) * (double)grid / w.sms + 0.5 * last);
    }
    return (double)((grid + w.sms - 1) / w.sms) * cta(item * std::max({std::ceil(items / cut.warps), items / cut.warps + 0.5, w.longest}));
}

/* `sms`: the part of the machine (`all`) this launch has when another runs beside it; `free_rows`: other rows than the rules'
 * may be tried. */
void balance_small(LaunchPlan* plan, const DeviceBatch& batch, const EvalProblem& prob, int sms, int all, Neighbour::Kind neighbour, size_t smem_limit,
                   bool free_rows) {
    const bool materialize = prob.mode == EVAL_MATERIALIZE;
    const uint32_t rr = (uint32_t)kVariantRows[plan->variant], rc = (uint32_t)kVariantBanks[plan->variant], pass = 32u * rr;
    const unsigned long long P = batch.num_programs, bank_groups = materialize ? 1 : (prob.num_banks + rc - 1) / rc;
    while (plan->perms_per_item > 1ull << batch.max_bits) plan->perms_per_item /= 2;
    /* as many warps as fit beside the tile buffers that are used */
    const auto refit = [&](LaunchPlan* p, uint32_t least) {
        const Geom g = make_geom(batch, prob, *p);
        const size_t tiles = (size_t)g.tile_bytes * g.tile_buffers + 16;
        p->warps = tiles < smem_limit ? (uint32_t)std::min<size_t>(20, (smem_limit - tiles) / g.warp_bytes) : 0u;
        p->warps = std::max(p->warps, least);
        p->smem_bytes = smem_needed(g, p->warps);
    };
    if (plan->tile_buffers == 1) refit(plan, plan->warps);
    /* a program has only as many values of its own as it reads toggle bits: the rules above counted all */
    const bool fewer = !materialize && batch.total_perms < 0.5 * (double)P * (double)(1ull << prob.toggle_bits);
    const unsigned long long rule_items = (P + plan->num_groups - 1) / plan->num_groups * (bank_groups / plan->groups_per_item);
    const unsigned long long rule_grid = (unsigned long long)plan->num_groups * plan->row_splits;
    /* deep enough, and its CTAs full enough; what is many waves of the whole machine is not confined to a part of it,
     * whose size is an estimate (358 programs, 33 sets, 770,512 rows, approximate functions: 6.9 ms, 10.3 when it was) */
    if (!fewer && rule_grid >= 8ull * (unsigned long long)sms && (rule_items >= 4ull * plan->warps || rule_grid >= 8ull * (unsigned long long)all)) return;
    /* what a pass of the row preludes costs beside one of the main parts; with toggles an item runs the shared prelude once
     * for all its permutations, and the few slots that leaves on the average serve better */
    const double prelude = !batch.max_hoisted ? 0.0 : batch.main_cost && !prob.toggle_bits ? 330.0 * (double)batch.prelude_cost / (double)batch.main_cost : 120.0;
    Work work{P, bank_groups, materialize ? 1.0 : batch.total_perms / (double)P, materialize ? 1.0 : (double)(1ull << batch.max_bits), 0, prelude, sms,
              batch.total_cost ? std::min(3.0, std::max(1.0, (double)batch.max_cost * (double)P / (double)batch.total_cost)) : 1.0};
    const auto passes_of = [&](uint32_t tile_rows) { return (uint32_t)((std::min<size_t>(tile_rows, prob.num_rows) + pass - 1) / pass); };
    Cut best{plan->tile_rows, (uint32_t)((plan->rows_per_split + plan->tile_rows - 1) / plan->tile_rows), plan->row_splits, plan->warps,
             plan->groups_per_item, plan->perms_per_item, 1u, plan->num_groups};
    work.passes = passes_of(plan->tile_rows);
    double least = 0.97 * cut_cycles(best, work);
    if (neighbour == Neighbour::LEAVES && rule_grid > (unsigned long long)sms) least = 1e300; /* any cut of one wave instead */
    const Cut rules = best;
    LaunchPlan trial = *plan;
    const bool uneven = work.perms < work.most_perms;
    for (uint32_t half = 0; half < (free_rows ? 2u : 1u); ++half) { /* the rules' tile and one of half its rows */
        trial.tile_rows = half ? (rules.tile_rows / 2 + pass - 1) / pass * pass : rules.tile_rows;
        if (half && (trial.tile_rows == rules.tile_rows || trial.tile_rows < 256u)) break;
        work.passes = passes_of(trial.tile_rows);
        const unsigned long long tiles = (prob.num_rows + trial.tile_rows - 1) / trial.tile_rows;
        for (trial.tile_buffers = 1; trial.tile_buffers <= (tiles > 1 ? 2u : 1u); ++trial.tile_buffers)
            for (uint32_t gpi = rules.gpi; gpi >= 1; --gpi) {
                if (bank_groups % gpi) continue;
                for (uint32_t ppi = gpi == bank_groups ? rules.ppi : 1u; ppi >= 1; ppi /= 2) {
                    trial.groups_per_item = gpi;
                    trial.perms_per_item = ppi;
                    refit(&trial, 0u);
                    if (trial.warps < std::min(rules.warps, 12u)) continue;
                    const unsigned long long items = materialize ? 1ull : ((bank_groups / gpi) << batch.max_bits) / ppi;
                    const unsigned most_waves = neighbour == Neighbour::LEAVES && !uneven ? 1u : fewer ? 32u : 8u;
                    for (unsigned waves = uneven ? 0u : 1u; waves <= most_waves; waves += waves < 8 ? 1 : 4) {
                        const unsigned long long ctas = waves ? (unsigned long long)waves * sms : rules.groups * rules.splits;
                        Cut c{trial.tile_rows, (uint32_t)((tiles + ctas - 1) / ctas), 0, trial.warps, gpi, ppi, 1u, 0};
                        if (!free_rows) c.tiles_per_split = rules.tiles_per_split;
                        if (uneven) c.warps = rules.warps;
                        if ((c.tiles_per_split > 1) != (trial.tile_buffers > 1)) continue;
                        c.splits = (uint32_t)((tiles + c.tiles_per_split - 1) / c.tiles_per_split);
                        c.groups = std::max<unsigned long long>(1, std::min(ctas / c.splits, P));
                        for (c.parts = 1; c.parts <= (free_rows ? work.passes : 1u); c.parts *= 2) {
                            if (items * c.parts > 0xffffff00ull / ((P + c.groups - 1) / c.groups)) break;
                            const double t = cut_cycles(c, work);
                            if (t < least) { least = t; best = c; }
                        }
                        if (waves && c.groups == P && c.tiles_per_split == 1) break; /* more waves are the same cut */
                    }
                }
            }
    }
    plan->tile_rows = best.tile_rows;
    plan->tile_buffers = best.tiles_per_split > 1 ? 2u : 1u;
    plan->row_splits = best.splits;
    plan->rows_per_split = (size_t)best.tiles_per_split * best.tile_rows;
    plan->groups_per_item = best.gpi;
    plan->perms_per_item = best.ppi;
    plan->parts = best.parts;
    plan->num_groups = (uint32_t)best.groups;
    plan->grid_x = plan->num_groups * plan->row_splits;
    refit(plan, 0u);
}

/* Most floats for the totals of passes (256 MB).  A launch that needs more has 8.6e9 values of rows to compute, 13 ms at least,
 * and is of many waves by the rules unless its programs are few; below, the totals pay (1,000 programs x 64 sets x 60,000 rows,
 * 30 million of them: 6.6 ms, 7.0 with the rules' rows). */
constexpr unsigned long long kMostPassSums = 1ull << 26;

LaunchPlan plan_with_tile(const DeviceBatch& batch, const EvalProblem& prob, int sm_count, size_t smem_limit, size_t scratch_limit,
                          int variant, bool balance, const Neighbour& neighbour, const RowCut* joint) {
    LaunchPlan plan{};
    plan.ok = false;
    plan.overflow = false;
    plan.groups_per_item = 1;
    plan.perms_per_item = 1;
    plan.parts = 1;
    plan.variant = variant;
    const uint32_t rr = (uint32_t)kVariantRows[variant], rc = (uint32_t)kVariantBanks[variant];
    const uint32_t pass = 32u * rr;
    const uint32_t nq = std::max<uint32_t>(1u, quantities(prob));
    const bool materialize = prob.mode == EVAL_MATERIALIZE;
    const uint32_t P = batch.num_programs;
    if (!P || !prob.num_rows || sm_count <= 0) return plan;

    /* Queue items: an item covers up to sixteen bank groups of one permutation, so the bank part and
     * the row prelude of a program are amortised over them; it never straddles permutations (toggles
     * are patched per item).  Fewer groups per item when the constant table or the partial sums of
     * sixteen groups would crowd out the tile. */
    unsigned long long items_per_program = 1;
    if (!materialize) {
        const unsigned long long bank_groups = (prob.num_banks + rc - 1) / rc;
        unsigned long long gpi = std::min<unsigned long long>(bank_groups, 16);
        for (;; --gpi) {
            if (bank_groups % gpi) continue;
            if (gpi == 1 || (gpi * batch.max_cst * rc * 4 <= 2048 && gpi * nq * rc * 4 <= 2048)) break;
        }
        plan.groups_per_item = (uint32_t)gpi;
        if (prob.toggle_bits > 40 || (bank_groups / gpi) > (~0ull >> prob.toggle_bits)) { plan.overflow = true; return plan; }
        /* An item that holds every bank group of its permutation may go on to the next permutations, up
         * to sixteen (permutation, bank group) pairs within the same table and partial-sum budgets: the
         * program is fetched once for them and its toggle-free row prelude runs once per row pass. */
        unsigned long long ppi = 1;
        if (gpi == bank_groups)
            while (ppi * 2 * gpi <= 16 && ppi * 2 <= (1ull << prob.toggle_bits) && ppi * 2 * gpi * batch.max_cst * rc * 4 <= 2048 &&
                   ppi * 2 * gpi * nq * rc * 4 <= 2048)
                ppi *= 2;
        plan.perms_per_item = (uint32_t)ppi;
        items_per_program = ((bank_groups / gpi) << prob.toggle_bits) / ppi;
    }
    /* item ids are 32-bit and every warp draws one id past the end */
    const unsigned long long kMaxItems = 0xffffff00ull;
    if (items_per_program > kMaxItems) { plan.overflow = true; return plan; }

    /* Warps per CTA and rows per tile.  20 warps run at a 96-register budget; a tile of at least
     * 512 rows keeps the per-item set-up (program copy, toggle patches, bank part) small against
     * the row passes, so fewer warps are preferred over a smaller tile down to 256 rows. */
    static const uint32_t warp_list[] = {20, 16, 12, 8, 4, 2, 1, 0};
    const uint32_t widest_tile = 1024;
    const size_t rows_padded = (prob.num_rows + pass - 1) / pass * pass;
    const uint32_t floors[3] = {512u, 256u, pass};
    for (int attempt = 0; attempt < 3 && !plan.ok; ++attempt) {
        const size_t floor_rows = std::min<size_t>(std::max<uint32_t>(floors[attempt], pass), rows_padded);
        for (const uint32_t* w = warp_list; *w && !plan.ok; ++w) {
            for (uint32_t want = widest_tile; want >= pass; want /= 2) {
                size_t tile_rows = std::min<size_t>(std::max<uint32_t>(want, pass) / pass * pass, rows_padded);
                if (tile_rows < floor_rows) break;
                LaunchPlan trial = plan;
                trial.warps = *w;
                trial.tile_rows = (uint32_t)tile_rows;
                trial.tile_buffers = rows_padded > tile_rows ? 2u : 1u;
                trial.num_groups = 1;
                trial.row_splits = 1;
                trial.rows_per_split = prob.num_rows;
                const Geom g = make_geom(batch, prob, trial);
                const size_t need = smem_needed(g, trial.warps);
                if (need > smem_limit) continue;
                plan = trial;
                plan.smem_bytes = need;
                plan.ok = true;
                break;
            }
        }
    }
    if (!plan.ok) return plan;
    plan.ok = false;

    /* Programs per CTA: at least eight queue items per warp and tile.  Programs arrive sorted by
     * cost and group g takes programs g, g + num_groups, ..., so every CTA's queue runs from its
     * costliest item to its cheapest and the warps reach the end of a tile close together. */
    unsigned long long want_items = 8ull * plan.warps;
    unsigned long long per_cta = (want_items + items_per_program - 1) / items_per_program;
    per_cta = std::max<unsigned long long>(1, std::min<unsigned long long>(per_cta, P));
    unsigned long long groups = std::max<unsigned long long>(1, P / per_cta);
    groups = std::min<unsigned long long>(groups, (unsigned long long)sm_count * 16ull);
    /* keep a CTA's item count inside 32 bits */
    while (((P + groups - 1) / groups) * items_per_program > kMaxItems && groups < P) groups = std::min<unsigned long long>(P, groups * 2);
    if (((P + groups - 1) / groups) * items_per_program > kMaxItems) { plan.overflow = true; return plan; }
    plan.num_groups = (uint32_t)groups;

    /* Rows are split across CTAs until the grid is many waves deep: a CTA that walks every row of
     * a large dataset runs for seconds and the last partial wave of such CTAs leaves most of the GPU
     * idle.  Each split keeps at least four tiles unless the program groups alone cannot fill the GPU. */
    const size_t tiles = (prob.num_rows + plan.tile_rows - 1) / plan.tile_rows;
    size_t want_ctas = (size_t)sm_count * 16;
    size_t most = groups >= (unsigned long long)sm_count * 2ull ? std::max<size_t>(1, tiles / 4) : tiles;
    size_t splits = std::min<size_t>(most, (want_ctas + (size_t)groups - 1) / (size_t)groups);
    splits = std::max<size_t>(1, splits);
    if (groups * splits < (unsigned long long)sm_count) { /* a small run: fewer programs per CTA rather than idle SMs */
        groups = std::min<unsigned long long>(P, ((unsigned long long)sm_count + splits - 1) / splits);
        plan.num_groups = (uint32_t)groups;
    }
    /* constant tables: one float per entry and (padded bank, permutation) */
    const unsigned long long padded = materialize ? rc : ((unsigned long long)(prob.num_banks + rc - 1) / rc * rc) << batch.max_bits;
    if (batch.total_cst > (~0ull >> 3) / padded) { plan.overflow = true; return plan; }
    plan.table_elements = (size_t)(batch.total_cst * padded);
    const unsigned long long configs = (unsigned long long)prob.num_banks << prob.toggle_bits;
    if (!materialize && configs) { /* [split][program][quantity][configuration] floats of scratch, in what the tables leave of it */
        const unsigned long long per_split = (unsigned long long)P * nq;
        if (per_split > (~0ull >> 3) / configs) { plan.overflow = true; return plan; }
        const unsigned long long room = scratch_limit > plan.table_elements ? (scratch_limit - plan.table_elements) / 4 * 4 : 0;
        const unsigned long long fit = std::max<unsigned long long>(1, room / (per_split * configs));
        splits = (size_t)std::min<unsigned long long>(splits, fit);
    }
    const size_t tiles_per_split = (tiles + splits - 1) / splits;
    plan.rows_per_split = tiles_per_split * plan.tile_rows;
    plan.row_splits = (uint32_t)((prob.num_rows + plan.rows_per_split - 1) / plan.rows_per_split);
    if (tiles_per_split == 1) plan.tile_buffers = 1;
    const unsigned long long grid = groups * plan.row_splits;
    if (grid > 0x7fffffffull) { plan.overflow = true; return plan; }
    plan.grid_x = (uint32_t)grid;

    const RowCut own{plan.tile_rows, plan.rows_per_split};
    plan.rules[0] = joint ? joint[0] : own;
    plan.rules[1] = joint ? joint[1] : own;
    const unsigned long long room = scratch_limit > plan.table_elements + 3 ? scratch_limit - plan.table_elements - 3 : 0;
    const unsigned long long passes = (prob.num_rows + pass - 1) / pass;
    const bool keeps_passes = !prob.toggle_bits && (materialize || passes <= std::min(room, kMostPassSums) / std::max(1ull, configs) / nq / P);
    if (joint && !keeps_passes) return plan;
    /* behind a launch that fills the machine the rules' rows stay as well: the estimate knows nothing of the SMs that become
     * free one by one (4,000 programs x 16 sets x 30,000 rows, 188 of them heavy: 3.89 ms with them, 4.39 with the cut it
     * prefers; 2,048 x 64 x 131,072: 28.6 and 28.1) */
    if (balance)
        balance_small(&plan, batch, prob, std::max(1, (int)(sm_count * neighbour.share)), sm_count, neighbour.kind, smem_limit,
                      keeps_passes && neighbour.kind != Neighbour::FILLS);
    plan.pass_sums = !materialize && (joint || plan.parts > 1 || plan.tile_rows != own.tile_rows || plan.rows_per_split != own.rows_per_split);
    plan.partial_elements = 0;
    if (!materialize) {
        const unsigned long long n = (plan.pass_sums ? passes : plan.row_splits) * P;
        if (configs && n > (~0ull >> 3) / configs / nq) { plan.overflow = true; return plan; }
        plan.partial_elements = (size_t)(n * nq * configs);
    }
    plan.table_offset = plan.pass_sums || plan.row_splits > 1 ? (plan.partial_elements + 3) / 4 * 4 : 0; /* whole sums go to the output */
    plan.ok = true;
    return plan;
}

}  // namespace

namespace {
LaunchPlan plan_any_tile(const DeviceBatch& batch, const EvalProblem& prob, int sm_count, size_t smem_limit, size_t scratch_limit, bool balance,
                         const Neighbour& neighbour, const RowCut* rules) {
    /* register tile: 4 rows x 4 banks per thread, or 8 x 2 / 16 x 1 when there are fewer banks.  Up
     * to four banks take the 8 x 2 tile: three or four banks are then two bank groups, so the row
     * prelude serves two runs of the main part and computes each row's value twice instead of four
     * times (measured on 4 banks x 256 permutations: 10 % faster than one 4 x 4 group; with 16 banks
     * and more the 4 x 4 tile is as fast or faster).  A tile with more rows per thread stages more
     * rows per pass; when even one pass of a wide dataset does not fit shared memory, the tiles with
     * fewer rows are tried (their spare bank columns compute padding that is never written). */
    int variant = prob.num_banks > 4 ? 0 : prob.num_banks >= 2 ? 1 : 2;
    if (prob.mode == EVAL_MATERIALIZE) variant = 2;
    LaunchPlan plan{};
    for (; variant >= 0; --variant) {
        plan = plan_with_tile(batch, prob, sm_count, smem_limit, scratch_limit, variant, balance, neighbour, rules);
        if (plan.ok || plan.overflow) break;
    }
    return plan;
}
}  // namespace

LaunchPlan plan_launch(const DeviceBatch& batch, const EvalProblem& prob, int sm_count, size_t smem_limit, size_t scratch_limit, Neighbour neighbour,
                       const RowCut* rules) {
    return plan_any_tile(batch, prob, sm_count, smem_limit, scratch_limit, true, neighbour, rules);
}
LaunchPlan plan_rules(const DeviceBatch& batch, const EvalProblem& prob, int sm_count, size_t smem_limit, size_t scratch_limit) {
    return plan_any_tile(batch, prob, sm_count, smem_limit, scratch_limit, false, Neighbour{Neighbour::NONE, 1.0}, nullptr);
}

}  // namespace sb
