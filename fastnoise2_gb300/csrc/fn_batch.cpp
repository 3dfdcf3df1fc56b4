// fn_batch.cpp -- descriptor staging, graph capture and autotuning for the
// batched persistent launch (kernel in fn_kernels.cu).
#include "fn_batch.h"

#include "fn_jit.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <sstream>
#include <unordered_map>

#include "FastNoise/FastNoise_C.h"

namespace fn {

namespace {
size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
}  // namespace

uint32_t tiles_for(long long total, uint32_t tile_points)
{
    if (total <= 0) return 1;                      // one empty tile still finalises min/max
    return (uint32_t)((total + tile_points - 1) / tile_points);
}

uint64_t batch_signature(const std::vector<BatchItem>& items, const std::vector<uint64_t>& hashes)
{
    // multiset of (program, size class): independent of request order and of node addresses
    std::vector<uint64_t> keys;
    keys.reserve(items.size());
    for (size_t i = 0; i < items.size(); ++i) {
        int lg = 0;
        while ((1ll << lg) < items[i].args.total && lg < 62) ++lg;
        keys.push_back(hashes[i] * 0x9E3779B97F4A7C15ull ^ ((uint64_t)items[i].args.src << 60) ^ ((uint64_t)lg << 48));
    }
    std::sort(keys.begin(), keys.end());
    return fnv1a64(keys.data(), keys.size() * sizeof(uint64_t));
}

BatchRunner::BatchRunner() {}

BatchRunner::~BatchRunner()
{
    if (exec_) cudaGraphExecDestroy(exec_);
    if (graph_) cudaGraphDestroy(graph_);
    if (staged_) cudaEventDestroy(staged_);
    if (fork_) cudaEventDestroy(fork_);
    for (auto e : join_) cudaEventDestroy(e);
    for (auto a : aux_) cudaStreamDestroy(a);
    if (capture_stream_) cudaStreamDestroy(capture_stream_);
    if (d_buf_) cudaFree(d_buf_);
    if (h_buf_) cudaFreeHost(h_buf_);
}

bool BatchRunner::reserve(size_t n_req, size_t n_items)
{
    if (n_req <= cap_req_ && n_items <= cap_items_) return true;
    size_t req = std::max(n_req, std::max<size_t>(cap_req_ * 2, 64));
    size_t items = std::max(n_items, std::max<size_t>(cap_items_ * 2, 4096));
    size_t off_req = align_up(sizeof(BatchHeader), 256);
    size_t off_state = align_up(off_req + req * sizeof(BatchRequest), 256);
    size_t off_groups = align_up(off_state + req * sizeof(BatchState), 256);
    size_t off_items = align_up(off_groups + req * sizeof(BatchGroup), 256);
    size_t bytes = align_up(off_items + items * sizeof(uint2), 256);
    char* d = nullptr;
    char* h = nullptr;
    if (!cuda_ok(cudaMalloc(&d, bytes), "cudaMalloc(batch descriptors)")) return false;
    if (!cuda_ok(cudaMallocHost(&h, bytes), "cudaMallocHost(batch staging)")) { cudaFree(d); return false; }
    if (d_buf_) cudaFree(d_buf_);
    if (h_buf_) cudaFreeHost(h_buf_);
    d_buf_ = d; h_buf_ = h;
    cap_req_ = req; cap_items_ = items; cap_bytes_ = bytes;
    off_req_ = off_req; off_state_ = off_state; off_groups_ = off_groups; off_items_ = off_items;
    d_states_ = reinterpret_cast<BatchState*>(d_buf_ + off_state_);
    if (exec_) { cudaGraphExecDestroy(exec_); exec_ = nullptr; }   // kernel arguments changed: recapture
    if (graph_) { cudaGraphDestroy(graph_); graph_ = nullptr; }
    return true;
}

bool BatchRunner::ensure_aux(size_t n)
{
    if (!fork_ && !cuda_ok(cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming), "event")) return false;
    while (aux_.size() < n) {
        cudaStream_t st = nullptr;
        cudaEvent_t ev = nullptr;
        if (!cuda_ok(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking), "stream")) return false;
        if (!cuda_ok(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "event")) { cudaStreamDestroy(st); return false; }
        aux_.push_back(st);
        join_.push_back(ev);
    }
    return true;
}

cudaError_t BatchRunner::launch_group(size_t g, uint32_t smem, cudaStream_t stream)
{
    auto* hdr = reinterpret_cast<BatchHeader*>(d_buf_);
    auto* reqs = reinterpret_cast<BatchRequest*>(d_buf_ + off_req_);
    auto* items = reinterpret_cast<uint2*>(d_buf_ + off_items_);
    const Group& gr = groups_[g];
    if (!gr.jit) return launch_batch(hdr, reqs, d_states_, items, smem, gr.grid, 256, stream);
    BatchState* states = d_states_;
    BatchGroup* grp = reinterpret_cast<BatchGroup*>(d_buf_ + off_groups_) + g;
    void* params[] = {&hdr, &reqs, &states, &items, &grp};
    return cudaLaunchKernel((const void*)gr.jit, dim3((unsigned)gr.grid), dim3((unsigned)gr.threads), params, 0, stream);
}

// Several group kernels run concurrently: fork from `stream` onto the auxiliary
// streams (round robin), join back before anything later on `stream`.  Works the
// same inside a stream capture, where it becomes parallel graph branches.
bool BatchRunner::launch_groups(cudaStream_t stream, uint32_t smem)
{
    if (groups_.size() == 1) return cuda_ok(launch_group(0, smem, stream), "launch batch");
    // Two groups on one stream wait for each other, and which two follows from the order of the trees
    // in the batch: with 8 streams for the chunk mix's 16 groups a batch of 220 requests took 322 or
    // 363 us, of 100 191 or 205; with 16 319 and 190 (of 4096: 4560 and 4537).
    const size_t na = std::min<size_t>(groups_.size(), 16);
    if (!ensure_aux(na)) return false;
    if (!cuda_ok(cudaEventRecord(fork_, stream), "fork")) return false;
    for (size_t a = 0; a < na; ++a)
        if (!cuda_ok(cudaStreamWaitEvent(aux_[a], fork_, 0), "fork wait")) return false;
    for (size_t g = 0; g < groups_.size(); ++g)
        if (!cuda_ok(launch_group(g, smem, aux_[g % na]), "launch batch group")) return false;
    for (size_t a = 0; a < na; ++a) {
        if (!cuda_ok(cudaEventRecord(join_[a], aux_[a]), "join")) return false;
        if (!cuda_ok(cudaStreamWaitEvent(stream, join_[a], 0), "join wait")) return false;
    }
    return true;
}

int BatchRunner::launch_graph(cudaStream_t stream, size_t bytes, uint32_t smem)
{
    // Recapture when the launch shape (kernels, grids, dynamic shared memory)
    // changed; otherwise only the upload node is updated -- the kernel arguments
    // are the fixed buffer addresses, the work lists travel in the upload.
    if (exec_ && (graph_groups_ != groups_ || graph_smem_ != smem)) {
        cudaGraphExecDestroy(exec_);
        exec_ = nullptr;
        if (graph_) { cudaGraphDestroy(graph_); graph_ = nullptr; }
    }
    if (!exec_) {
        graph_groups_ = groups_;
        graph_smem_ = smem;
        copy_node_ = nullptr;
        if (!capture_stream_ && !cuda_ok(cudaStreamCreateWithFlags(&capture_stream_, cudaStreamNonBlocking), "stream")) return -3;
        if (!cuda_ok(cudaStreamBeginCapture(capture_stream_, cudaStreamCaptureModeThreadLocal), "begin capture")) return -3;
        cudaMemcpyAsync(d_buf_, h_buf_, bytes, cudaMemcpyHostToDevice, capture_stream_);
        const bool queued = launch_groups(capture_stream_, smem);
        cudaGraph_t g = nullptr;
        const bool ended = cuda_ok(cudaStreamEndCapture(capture_stream_, &g), "end capture");
        if (!queued || !ended) { if (g) cudaGraphDestroy(g); return -3; }
        graph_ = g;
        if (!cuda_ok(cudaGraphInstantiate(&exec_, graph_, 0), "graph instantiate")) return -3;
        size_t n = 0;
        cudaGraphGetNodes(graph_, nullptr, &n);
        std::vector<cudaGraphNode_t> nodes(n);
        cudaGraphGetNodes(graph_, nodes.data(), &n);
        for (auto nd : nodes) {
            cudaGraphNodeType t;
            cudaGraphNodeGetType(nd, &t);
            if (t == cudaGraphNodeTypeMemcpy) copy_node_ = nd;
        }
        if (!copy_node_) { set_error(-3, "unexpected graph shape"); return -3; }
    } else {
        if (!cuda_ok(cudaGraphExecMemcpyNodeSetParams1D(exec_, copy_node_, d_buf_, h_buf_, bytes, cudaMemcpyHostToDevice), "graph memcpy update"))
            return -3;
    }
    return cuda_ok(cudaGraphLaunch(exec_, stream), "graph launch") ? 0 : -3;
}

int BatchRunner::launch(const std::vector<BatchItem>& items, cudaStream_t stream, const BatchTuning* tuning_in, bool use_graph)
{
    const size_t n = items.size();
    if (n == 0) return 0;
    // A batch has few trees: each is looked up once, not once per request.
    struct Tree {
        DeviceProgram prog;
        BatchKernel kernel;            // its specialised batch kernel
        JitKernels jk;                 // its column kernel
        int group[2] = {-1, -1};       // launch group of its point / column requests
        // its requests that can be walked in columns: microseconds of each route, what columns save
        // over those that gain and lose over the others, and the 32-point steps
        double point_us = 0, column_us = 0, won = 0, lost = 0;
        double work = 0, gain_work = 0;
        long long largest = 0;         // points of the largest
        unsigned longest = 0;          // steps of the longest unit
        float step_us = 0, enter_us = 0;
        enum Walk : char { kPoints, kGains, kColumns } plan = kPoints, walk = kPoints;   // kGains: those that gain
        // the estimates of its last grid shapes: a batch's requests have few (100 ns each otherwise)
        struct Estimate {
            int count[4];
            float step[4];
            bool column;
            ColumnShape shape;
            float point_us, column_us;
        };
        std::vector<Estimate> estimates;
        size_t next_estimate = 0;
    };
    std::vector<Tree> trees;
    std::unordered_map<uintptr_t, uint32_t> tree_index;
    tree_of_.resize(n);
    uint32_t max_bytes = 16;
    points_ = 0;
    bool jit = true;
    for (size_t i = 0; i < n; ++i) {
        const BatchItem& it = items[i];
        if (!it.node || it.args.total < 0 || (it.args.total > 0 && !it.dout)) {
            set_error(-1, "batch request " + std::to_string(i) + ": invalid arguments");
            return -1;
        }
        const auto known = tree_index.emplace(reinterpret_cast<uintptr_t>(it.node) * 8 + (uintptr_t)it.args.dim, (uint32_t)trees.size());
        if (known.second) {
            trees.emplace_back();
            DeviceProgram& prog = trees.back().prog;
            if (!get_program(it.node, it.args.dim, prog)) return last_error();
            std::string err;
            if (!jit_ensure(prog.host, err)) { set_error(-2, "batch request " + std::to_string(i) + ": " + err); return -2; }
            max_bytes = std::max(max_bytes, prog.bytes);
        }
        tree_of_[i] = known.first->second;
        points_ += (uint64_t)it.args.total;
        jit = jit && it.args.total < (1ll << 32);   // 32-bit point indices
    }
    // Specialised batch kernels when every program of the batch has one: each tree's tuned
    // variant when it is built (a variant not built yet is queued for a background build and
    // variant 0 runs meanwhile).
    for (size_t t = 0; jit && t < trees.size(); ++t) {
        Tree& tr = trees[t];
        const uint64_t hash = tr.prog.hash;
        const int v = Autotuner::instance().tree_variant(hash);
        bool ok = jit_batch_kernel(hash, v, tr.kernel);
        if (!ok && !jit_is_specialised(hash) && jit_try_cached(tr.prog.host))   // an earlier process built it
            ok = jit_batch_kernel(hash, v, tr.kernel);
        if (!ok && v != 0) {
            jit_request_batch_variants(tr.prog.host);
            ok = jit_batch_kernel(hash, 0, tr.kernel);
        }
        if (!ok) { jit = false; break; }
        if (!jit_lookup(hash, tr.jk)) tr.jk = JitKernels();
    }
    if (!jit)                                       // interpreter batch: count a use of each program
        for (size_t t = 0; t < trees.size(); ++t) {
            bool seen = false;
            for (size_t u = 0; u < t; ++u) seen = seen || trees[u].prog.hash == trees[t].prog.hash;
            if (!seen) jit_note_interpreted(trees[t].prog.host);
        }
    if (!jit)
        for (size_t i = 0; i < n; ++i)
            if (trees[tree_of_[i]].prog.host->needs_specialisation() && items[i].args.total > 0) {
                set_error(-2, "batch request " + std::to_string(i) + ": the tree needs specialised kernels, which this batch "
                              "cannot use (specialisation disabled or a request of 2^32 points or more)");
                return -2;
            }
    // the signature sorts a key per request: only for a tuning run, or to look one up
    signature_ = 0;
    if (tuning_in || Autotuner::instance().any()) {
        std::vector<uint64_t> hashes;
        for (uint32_t t : tree_of_) hashes.push_back(trees[t].prog.hash);
        signature_ = batch_signature(items, hashes);
        if (jit) signature_ = signature_ * 0x100000001B3ull + 0x4A17;   // tuned separately from the interpreter
    }
    BatchTuning tuning;
    if (tuning_in) tuning = *tuning_in;
    else Autotuner::instance().lookup(signature_, tuning);
    const uint32_t tp = std::max<uint32_t>(256, tuning.tile_points);
    columns_.assign(n, ColumnShape());
    saved_.assign(n, 0.0f);
    for (size_t i = 0; jit && i < n; ++i) {
        Tree& tr = trees[tree_of_[i]];
        const PointArgs& a = items[i].args;
        if (a.src != kSrcGrid) continue;
        const Tree::Estimate* e = nullptr;
        for (const Tree::Estimate& k : tr.estimates)
            if (!std::memcmp(k.count, a.count, sizeof k.count) && !std::memcmp(k.step, a.step, sizeof k.step)) { e = &k; break; }
        if (!e) {
            if (tr.estimates.size() < 8) tr.estimates.emplace_back();
            Tree::Estimate& k = tr.estimates[tr.next_estimate++ % 8];
            std::memcpy(k.count, a.count, sizeof k.count);
            std::memcpy(k.step, a.step, sizeof k.step);
            k.column = jit_batch_columns(a, tr.jk, k.shape, k.point_us, k.column_us);
            e = &k;
        }
        if (!e->column) continue;
        columns_[i] = e->shape;
        saved_[i] = e->point_us - e->column_us;
        const double work = (double)e->shape.steps * column_chunks(e->shape);
        tr.point_us += e->point_us;
        tr.column_us += e->column_us;
        (saved_[i] > 0.0f ? tr.won : tr.lost) += saved_[i];
        tr.work += work;
        if (saved_[i] > 0.0f) tr.gain_work += work;
        tr.largest = std::max(tr.largest, (long long)a.total);
        tr.longest = std::max(tr.longest, (unsigned)std::min(64.0, std::ceil(work / 8.0)));
        tr.step_us = std::max(tr.step_us, e->shape.step_us);
        tr.enter_us = std::max(tr.enter_us, e->shape.enter / 3000.0f);
    }
    // Column units: about four rounds of 16 warps per SM over the whole batch, so that short
    // batches still spread, and at most 64 steps (longer ones gain under 5 % of set-up).
    auto unit_steps = [](double work) { return (unsigned)std::min(64.0, std::max(4.0, work / (64.0 * num_sms()))); };
    // Which grid requests are walked in columns: none, those of the trees that issue less so, or all
    // that can be.  A batch of one tree takes what its requests issue, and not less than its longest
    // tile, whose threads take their points one after another, or its longest unit, whose warp takes
    // its steps so; columns add 3 us, a longer first step and last units.  Large batches are decided by
    // what they issue, small ones by the longest tile or unit: 4 requests of terrain 32^3 59 us as
    // points, 28 in columns, of CellularValue 45 / 21; 106 of FBm(Perlin) 34 x 47 25 / 36.
    //
    // Several trees are decided by what they issue, and have to gain 6 us.  The longest tile would often
    // speak for columns there too (8 requests of 8 trees, 40 000 points, 58 / 32 us), but a server's
    // batches of that size then end before the next is submitted, and no longer run beside each other.
    //
    // A tree's requests stay together unless those that would lose lose more than a second group costs
    // (the 155 smallest 2D grids of the 4096-request chunk mix: split off 4840 us, together 4550).
    constexpr double kGroupUs = 10.0, kPointUs = 1.0 / 500.0;   // a warp's points: us per issue slot
    const bool one = trees.size() == 1;
    const double columns_us = one ? 3.0 : 6.0;
    double best_us = 1e30;
    for (int plan = 0; plan < 3; ++plan) {
        if (grid_route().route == FN_GRID_ROUTE_COLUMNS && plan < 2) continue;
        double issue = 0, chain = 0, work = 0;
        for (Tree& tr : trees) {
            tr.plan = plan == 2 ? Tree::kColumns : Tree::kPoints;
            if (plan == 1 && tr.lost < -kGroupUs && tr.won > 0.0) tr.plan = Tree::kGains;
            else if (plan == 1 && tr.won + tr.lost > 0.0) tr.plan = Tree::kColumns;
            issue += tr.plan == Tree::kPoints ? tr.point_us : tr.plan == Tree::kGains ? tr.point_us - tr.won : tr.column_us;
            work += tr.plan == Tree::kPoints ? 0.0 : tr.plan == Tree::kGains ? tr.gain_work : tr.work;
        }
        const unsigned len = unit_steps(work);
        for (const Tree& tr : trees) {
            if (!one) break;
            if (tr.plan != Tree::kColumns)
                chain = std::max(chain, (double)((std::min<long long>(tr.largest, tp) + 255) / 256) * tr.jk.point_cost * kPointUs);
            if (tr.plan != Tree::kPoints) chain = std::max(chain, (double)(std::min(len, tr.longest) * tr.step_us + tr.enter_us));
        }
        const double us = std::max(issue, chain) + (plan ? columns_us : 0.0);
        if (us >= best_us) continue;
        best_us = us;
        for (Tree& tr : trees) tr.walk = tr.plan;
    }
    double column_work = 0;
    for (size_t i = 0; i < n; ++i) {
        const Tree& tr = trees[tree_of_[i]];
        if (tr.walk == Tree::kPoints || (tr.walk == Tree::kGains && !(saved_[i] > 0.0f))) columns_[i] = ColumnShape();
        if (!columns_[i].plane) continue;
        column_work += (double)columns_[i].steps * column_chunks(columns_[i]);
        ++grid_route().columns;
    }
    const unsigned col_len = unit_steps(column_work);
    // One group per distinct kernel, in first-appearance order (the interpreter: one for all).
    std::vector<BatchKernel> gkernel;
    std::vector<char> gcolumn;                      // whether it walks columns
    std::vector<size_t> gitems;                     // work items per group
    tiles_.resize(n);
    group_of_.resize(n);
    size_t n_items = 0;
    for (size_t i = 0; i < n; ++i) {
        const bool column = columns_[i].plane != 0;
        tiles_[i] = column ? column_tiles(columns_[i], col_len) : tiles_for(items[i].args.total, tp);
        Tree& tr = trees[tree_of_[i]];
        int& g = tr.group[column ? 1 : 0];
        if (g < 0) {
            const BatchKernel bk = !jit ? BatchKernel{nullptr, 256} : column ? BatchKernel{tr.jk.batch_column, 256} : tr.kernel;
            for (g = 0; g < (int)gkernel.size() && gkernel[(size_t)g].kernel != bk.kernel; ++g) {}
            if (g == (int)gkernel.size()) {
                gkernel.push_back(bk);
                gcolumn.push_back(column);
                gitems.push_back(0);
            }
        }
        group_of_[i] = (uint32_t)g;
        gitems[(size_t)g] += tiles_[i];
        n_items += tiles_[i];
    }
    if (n_items > 0xFFFFFFFFull) { set_error(-4, "batch too large"); return -4; }
    point_trees_.clear();
    for (const Tree& tr : trees)
        if (tr.group[0] >= 0) point_trees_.push_back(tr.prog.hash);
    if (!reserve(n, n_items)) return -3;

    // The staging buffer is reused: the previous launch's upload must have been consumed.
    if (!staged_ && !cuda_ok(cudaEventCreateWithFlags(&staged_, cudaEventDisableTiming), "event")) return -3;
    cudaEventSynchronize(staged_);

    auto* hdr = reinterpret_cast<BatchHeader*>(h_buf_);
    auto* reqs = reinterpret_cast<BatchRequest*>(h_buf_ + off_req_);
    auto* states = reinterpret_cast<BatchState*>(h_buf_ + off_state_);
    auto* grps = reinterpret_cast<BatchGroup*>(h_buf_ + off_groups_);
    auto* its = reinterpret_cast<uint2*>(h_buf_ + off_items_);
    std::memset(hdr, 0, sizeof(BatchHeader));
    hdr->n_req = (unsigned)n;
    hdr->n_items = (unsigned)n_items;
    hdr->tile_points = tp;
    hdr->max_prog_bytes = max_bytes;
    last_minmax_.resize(n);
    for (size_t i = 0; i < n; ++i) {
        BatchRequest& r = reqs[i];
        std::memset(&r, 0, sizeof r);
        const DeviceProgram& prog = trees[tree_of_[i]].prog;
        r.args = items[i].args;
        if (columns_[i].plane) column_args(r.args, columns_[i]);
        r.prog = prog.dptr;
        r.jit_slot = -1;
        r.prog_bytes = prog.bytes;
        r.out = items[i].dout;
        r.minmax = items[i].dminmax;
        r.host_minmax = items[i].host_minmax;
        r.host_done = items[i].host_done;
        r.host_time = items[i].host_time;
        r.n_tiles = tiles_[i];
        states[i].mn_enc = 0xFFFFFFFFu;
        states[i].mx_enc = 0u;
        states[i].tiles_done = 0u;
        states[i].pad = 0u;
        last_minmax_[i] = items[i].dminmax;
    }
    const int sms = num_sms();
    groups_.assign(gkernel.size(), Group());
    std::vector<size_t> next(gkernel.size());       // next item of each group
    for (size_t g = 0, k = 0; g < gkernel.size(); ++g) {
        next[g] = k;
        k += gitems[g];
    }
    int total_grid = 0;
    for (size_t g = 0; g < gkernel.size(); ++g) {
        Group& gr = groups_[g];
        gr.jit = gkernel[g].kernel;
        gr.threads = gkernel[g].threads;
        gr.item_begin = (uint32_t)next[g];
        gr.item_end = (uint32_t)(next[g] + gitems[g]);
        grps[g].item_begin = gr.item_begin;
        grps[g].item_end = gr.item_end;
        grps[g].head = 0;
        grps[g].pad = 0;
        // A tuned number of CTAs goes with the tuned tile size: column groups, whose items are cut
        // otherwise, take what fits on an SM.
        int occ = gcolumn[g] ? 0 : tuning.ctas_per_sm;
        if (occ <= 0 && gr.jit) {
            int& known = occupancy_[gr.jit];
            if (!known && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&known, (const void*)gr.jit, gr.threads, 0) != cudaSuccess || known < 1))
                known = 1;
            occ = known;
        } else if (occ <= 0) {
            occ = batch_occupancy(256, max_bytes);
        }
        long long grid = (long long)sms * occ;
        const long long group_items = (long long)(gr.item_end - gr.item_begin);
        if (grid > group_items) grid = group_items;
        if (grid < 1) grid = 1;
        gr.grid = (int)grid;
        total_grid += gr.grid;
    }
    for (size_t i = 0; i < n; ++i) {
        uint2* at = its + next[group_of_[i]];
        for (uint32_t t = 0; t < tiles_[i]; ++t) at[t] = make_uint2((unsigned)i, t);
        next[group_of_[i]] += tiles_[i];
    }
    const size_t bytes = off_items_ + n_items * sizeof(uint2);
    const uint32_t smem = jit ? 0 : max_bytes;
    // A graph pays off for a launch shape that repeats (the same batch every frame); batches
    // whose shape keeps changing (a server's admissions) would pay a capture each time, so a
    // new shape is captured only when it comes twice in a row and runs as plain launches until then.
    const bool same_as_graph = exec_ && graph_groups_ == groups_ && graph_smem_ == smem;
    const bool repeated = last_groups_ == groups_ && last_smem_ == smem;
    last_groups_ = groups_;
    last_smem_ = smem;
    int rc;
    if (use_graph && (same_as_graph || repeated)) {
        rc = launch_graph(stream, bytes, smem);
    } else {
        rc = cuda_ok(cudaMemcpyAsync(d_buf_, h_buf_, bytes, cudaMemcpyHostToDevice, stream), "upload batch") &&
                     launch_groups(stream, smem)
                 ? 0
                 : -3;
    }
    if (rc == 0) {
        cudaEventRecord(staged_, stream);
        items_ = n_items;
        upload_bytes_ = bytes;
        tile_points_ = tp;
        grid_ = total_grid;
        specialised_ = jit;
    }
    return rc;
}

// ------------------------------------------------------------------ autotuner

Autotuner& Autotuner::instance()
{
    static Autotuner a;
    return a;
}

bool Autotuner::lookup(uint64_t sig, BatchTuning& out)
{
    std::lock_guard<std::mutex> lk(mu_);
    auto it = table_.find(sig);
    if (it == table_.end()) return false;
    out = it->second.first;
    return true;
}

bool Autotuner::any()
{
    std::lock_guard<std::mutex> lk(mu_);
    return !table_.empty();
}

void Autotuner::store(uint64_t sig, const BatchTuning& t, double ms)
{
    std::lock_guard<std::mutex> lk(mu_);
    auto it = table_.find(sig);
    if (it == table_.end() || ms < it->second.second) table_[sig] = {t, ms};
}

std::vector<BatchTuning> Autotuner::candidates() const
{
    std::vector<BatchTuning> c;
    for (uint32_t tp : {1024u, 2048u, 4096u, 8192u})
        for (int ctas : {0, 1}) c.push_back(BatchTuning{tp, ctas});
    return c;
}

int Autotuner::tree_variant(uint64_t program_hash)
{
    std::lock_guard<std::mutex> lk(mu_);
    auto it = trees_.find(program_hash);
    return it == trees_.end() ? 0 : it->second.first;
}

bool Autotuner::tree_tuned(uint64_t program_hash)
{
    std::lock_guard<std::mutex> lk(mu_);
    return trees_.count(program_hash) != 0;
}

void Autotuner::store_tree(uint64_t program_hash, int variant, double ms)
{
    std::lock_guard<std::mutex> lk(mu_);
    trees_[program_hash] = {variant, ms};
}

// Text format, one entry per line:
//   <signature hex> <tile points> <CTAs per SM> <ms>                         a batch signature
//   tree <program hash hex> <variant> <threads> <blocks per SM> <points> <ms>  a tree's batch kernel
bool Autotuner::load(const std::string& path)
{
    std::ifstream f(path);
    if (!f) return false;
    std::lock_guard<std::mutex> lk(mu_);
    std::string line;
    while (std::getline(f, line)) {
        std::istringstream in(line);
        std::string first;
        if (!(in >> first)) continue;
        if (first == "tree") {
            unsigned long long hash;
            int variant, threads, blocks, points;
            double ms;
            if (in >> std::hex >> hash >> std::dec >> variant >> threads >> blocks >> points >> ms && variant >= 0 &&
                (size_t)variant < batch_variants().size())
                trees_[hash] = {variant, ms};
        } else {
            unsigned long long sig = std::strtoull(first.c_str(), nullptr, 16);
            unsigned tp;
            int ctas;
            double ms;
            if (in >> tp >> ctas >> ms) table_[sig] = {BatchTuning{tp, ctas}, ms};
        }
    }
    return true;
}

bool Autotuner::save(const std::string& path) const
{
    std::ofstream f(path);
    if (!f) return false;
    for (const auto& kv : table_)
        f << std::hex << kv.first << std::dec << ' ' << kv.second.first.tile_points << ' ' << kv.second.first.ctas_per_sm << ' '
          << kv.second.second << '\n';
    for (const auto& kv : trees_) {
        const BatchVariant& v = batch_variants()[(size_t)kv.second.first];
        f << "tree " << std::hex << kv.first << std::dec << ' ' << kv.second.first << ' ' << v.threads << ' ' << v.min_blocks << ' '
          << v.points << ' ' << kv.second.second << '\n';
    }
    return true;
}

}  // namespace fn
