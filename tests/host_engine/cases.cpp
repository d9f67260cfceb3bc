// The engine's host code on the CPU: engine.cu and hostcopy.cu over the CUDA
// runtime beside this file, with kernels that only leave the counts which the
// host reads.  Each case makes a call fail and returns 0 when the engine says so.
#include "../../empanada_b200/csrc/engine.cu"
#include "../../empanada_b200/csrc/hostcopy.cu"

#include <thread>

namespace fake {
// a set has so many reads per parse tile of its FASTQ, three read-ends in four unique
constexpr uint64_t kReads = 100, kLen = 50;
uint64_t reads(uint64_t F) { return kReads * emp::parse_tiles(F); }
std::function<void(uint32_t *err)> on_init_list;
std::function<void(emp::SweepJob &)> on_sweep;
std::function<cudaError_t()> on_bucket;
int graph_builds = 0;
bool sort_buffers = false;
}  // namespace fake

namespace emp {
void launch_nl_count(const uint8_t *, uint64_t, uint32_t *, uint64_t *, cudaStream_t) {}
void launch_scan_u32_u64(const uint32_t *, uint64_t *, uint64_t n, uint64_t *, uint32_t *, uint64_t *total, uint32_t *,
                         cudaStream_t) {
    *total = 4 * fake::kReads * n;
}
void launch_scan_u32_u32(const uint32_t *, uint32_t *, uint64_t, uint64_t *, uint32_t *, uint64_t *, uint32_t *,
                         cudaStream_t) {}
void launch_nl_count_many(const NlArgs *, ManyBlocks, cudaStream_t) {}
void launch_scan_many(const ScanArgs *a, ManyBlocks b, cudaStream_t) {
    for (uint32_t i = 0; i < b.n; ++i) *a[b.blk[i].x].total = 4 * fake::kReads * a[b.blk[i].x].n;
}
void launch_read_pass_many(const ReadArgs *a, ManyBlocks b, cudaStream_t) {
    for (uint32_t i = 0; i < b.n; ++i) {
        const ReadArgs &x = a[b.blk[i].x];
        *x.n_kept = fake::reads(x.F);
        x.len_minmax[0] = ~(uint32_t)fake::kLen;
        x.len_minmax[1] = fake::kLen;
    }
}
uint32_t read_pass_grid() { return 148; }
void launch_dedup_many(const DedupArgs *, uint32_t, uint32_t, ManyBlocks, ManyBlocks, ManyBlocks, cudaStream_t) {}
void launch_init_list_many(const InitArgs *, ManyBlocks, cudaStream_t) {}
void launch_upload(const void *host, void *dev, size_t bytes, cudaStream_t) { std::memcpy(dev, host, bytes); }
void launch_gather_words(const uint64_t *const *src, uint32_t jobs, uint64_t *out, cudaStream_t) {
    for (uint32_t k = 0; k < jobs; ++k) std::memcpy(out + 16 * k, src[k], 128);
}
void launch_read_pass(const uint8_t *, uint64_t F, const uint64_t *, const HashTables *, const ChunkWeights *, uint64_t *,
                      uint32_t *, int, uint32_t *, uint64_t *n_kept, uint32_t *len_minmax, uint32_t *, cudaStream_t) {
    *n_kept = fake::reads(F);
    len_minmax[0] = ~(uint32_t)fake::kLen;
    len_minmax[1] = fake::kLen;
}
void launch_compact_reads(const uint32_t *, uint64_t, uint64_t, const uint64_t *, const uint32_t *, int, uint64_t *,
                          uint32_t *, cudaStream_t) {}
void launch_columns(const uint32_t *, uint64_t, int, int, uint32_t *, uint64_t, cudaStream_t) {}
uint32_t dedup_buckets(uint64_t) { return 1; }
bool dedup_args(DedupArgs *, const uint64_t *, uint64_t, uint32_t, void *, uint64_t *, uint32_t *, uint8_t *,
                uint32_t *) { return false; }
bool launch_dedup_hash(const uint64_t *, uint64_t, uint32_t, void *, uint64_t *, uint32_t *, uint8_t *, uint32_t *,
                       cudaStream_t) { return true; }
void launch_dedup_mark(const uint64_t *, const uint32_t *, uint64_t, uint8_t *, cudaStream_t) {}
void launch_init_list(const uint64_t *, const uint8_t *, uint64_t n, uint64_t *, uint32_t *, uint64_t *, uint32_t *,
                      uint64_t *count, uint32_t *err, cudaStream_t) {
    *count = 2 * n * 3 / 4;
    if (fake::on_init_list) fake::on_init_list(err);
}
void launch_dup_prefix_half(uint64_t *, uint32_t *, uint64_t, cudaStream_t) {}
void launch_iota(uint32_t *, uint64_t, cudaStream_t) {}
void launch_update_compact(const RoundArgs &, cudaStream_t) {}
void launch_split_tables(const uint64_t *, const uint32_t *, uint64_t, uint64_t *, uint32_t *, uint64_t *, uint64_t *,
                         uint32_t *, uint32_t *, cudaStream_t) {}
void launch_search_partitions(const uint64_t *, uint64_t, const uint64_t *, uint64_t, uint64_t, const uint32_t *,
                              const uint64_t *, uint64_t, SearchPart *, uint64_t, uint64_t *, uint64_t *, uint32_t *,
                              cudaStream_t) {}
void launch_write_records(const SearchPart *, uint64_t, uint64_t, int32_t, const uint32_t *, const uint32_t *, uint8_t *,
                          cudaStream_t) {}
void launch_join_count(const uint64_t *, const uint32_t *, uint64_t, uint32_t *, cudaStream_t) {}
void launch_join_write(const uint64_t *, const uint32_t *, uint64_t, const uint32_t *, const uint64_t *, uint32_t *,
                       uint32_t *, uint8_t *, uint8_t *, cudaStream_t) {}
void launch_chunk_keys(const uint32_t *, uint64_t, const uint32_t *, uint64_t, int, uint64_t *, uint32_t *,
                       cudaStream_t) {}
void launch_ring_gather(const uint64_t *, const uint32_t *, const uint32_t *, uint64_t, uint64_t *, uint32_t *,
                        cudaStream_t) {}
void launch_ring_copy(const uint64_t *, const uint32_t *, uint64_t, uint64_t, uint64_t, uint64_t *, uint32_t *,
                      cudaStream_t) {}
void launch_merge(uint64_t *, uint32_t *, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t,
                  ChunkPart *, uint64_t, uint64_t *, uint32_t *, cudaStream_t) {}
void launch_unique_walk(const uint64_t *, uint64_t, uint64_t, uint32_t *, cudaStream_t) {}

size_t sort_scratch_bytes(uint64_t) { return 4096; }
void sort_pairs(uint64_t *, uint32_t *, uint64_t *, uint32_t *, uint64_t, void *, uint32_t *, cudaStream_t,
                cudaEvent_t *) {}
void sort_groups(uint64_t *, uint32_t *, uint64_t *k1, uint32_t *v1, uint64_t, void *scratch, uint32_t *, cudaStream_t) {
    fake::sort_buffers = k1 && v1 && scratch;
}
void sort_radix(uint64_t *, uint32_t *, uint64_t *, uint32_t *, uint64_t, void *, uint32_t *, cudaStream_t,
                cudaEvent_t *) {}
int sort_moves(uint64_t) { return 1; }
uint32_t *sort_flags(void *p) { return static_cast<uint32_t *>(p); }
void sort_top_digit(const uint64_t *, const uint32_t *, uint64_t *, uint32_t *, uint64_t, void *, uint32_t *,
                    cudaStream_t) {}

int bucket_grid_size() { return 148; }
size_t bkt_scratch_bytes(uint64_t) { return 4096; }
cudaError_t launch_bucket_rounds(BktJob *jobs, CoopCtl *ctl, uint32_t *, cudaStream_t) {
    for (uint32_t k = 0; k < ctl->njobs; ++k) {
        jobs[k].done = 1;
        jobs[k].round = (uint32_t)jobs[k].r0;
    }
    return fake::on_bucket ? fake::on_bucket() : cudaSuccess;
}
cudaError_t launch_bucket_list(BktJob *, uint64_t *, uint32_t *, cudaStream_t) { return cudaSuccess; }
bool bucket_prologue_apart(const BktJob &) { return false; }
cudaError_t launch_bucket_prologue(BktJob *, cudaStream_t) { return cudaSuccess; }
cudaError_t measure_l2_read(uint64_t, double *) { return cudaSuccess; }

int sweep_grid_size() { return 148; }
uint32_t sweep_segment_size(uint64_t) { return 32; }
uint32_t sweep_first_rounds(uint64_t, uint64_t) { return 4; }
uint32_t sweep_shard_log(uint64_t, uint64_t) { return 0; }
uint32_t sweep_bins_max(uint64_t, int) { return 64; }
size_t sweep_layout(uint8_t *, SweepJob *, size_t *zeroed) { return *zeroed = 4096; }
size_t sweep_out_layout(uint8_t *, uint32_t, SweepOut *, size_t *zeroed) { return *zeroed = 4096; }
cudaError_t launch_sweep(SweepJob *jobs, CoopCtl *ctl, const SweepOut &, bool, cudaStream_t) {
    for (uint32_t k = 0; k < ctl->njobs; ++k) {
        jobs[k].round = (uint32_t)jobs[k].r0;
        if (fake::on_sweep) fake::on_sweep(jobs[k]);
    }
    return cudaSuccess;
}

void graph_paths(const uint8_t *, const uint64_t *, const uint64_t *, uint32_t, uint64_t, uint32_t, const GraphBufs &,
                 cudaStream_t) { ++fake::graph_builds; }
void graph_cycles(uint32_t, const GraphBufs &, cudaStream_t) {}
void graph_place(uint32_t nodes, const GraphBufs &b, cudaStream_t) {  // every read-end a unitig of its own
    for (uint32_t u = 0; u < nodes; ++u) {
        b.order[u] = u;
        b.starts[u] = u;
    }
    b.total[0] = b.total[1] = nodes;
}
}  // namespace emp

// a host allocation of this thread that fails: the n-th from now
static thread_local int alloc_countdown = 0;
void *operator new(size_t n) {
    if (alloc_countdown > 0 && --alloc_countdown == 0) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

namespace {

emp_ctx *make_ctx(uint64_t budget = 0) {
    emp_ctx *c = nullptr;
    if (emp_ctx_create(0, budget, &c) != EMP_OK) std::abort();
    return c;
}
emp_job *fed_job(emp_ctx *c, uint64_t bytes = 10000) {
    emp_params p;
    emp_params_default(&p);
    emp_job *j = nullptr;
    const std::string fq(bytes, 'A');
    if (emp_job_create(c, &p, &j) != EMP_OK || emp_job_feed_fastq(j, fq.data(), fq.size(), 1) != EMP_OK) std::abort();
    return j;
}

// The list built again for a larger edge buffer: a look-back of it that runs
// out of its wait is the run's status.
int rebuilt_list_times_out() {
    emp_ctx *c = make_ctx();
    emp_job *j = fed_job(c);
    int sweeps = 0, lists = 0;
    fake::on_sweep = [&](emp::SweepJob &x) {
        x.overflow = ++sweeps == 1;
        x.e_total = x.ecap + 1;
    };
    if (emp_job_run(j, nullptr) != EMP_OK || sweeps != 2) return 1;
    sweeps = 0;
    fake::on_init_list = [&](uint32_t *err) {
        if (++lists == 2) *err |= emp::kErrSpin;
    };
    const emp_status st = emp_job_run(j, nullptr);
    if (lists != 2) return 2;
    return st == EMP_E_TIMEOUT ? 0 : 3;
}

// output.bin bytes of one record with n edges between the first two read-ends
std::vector<uint8_t> one_record(uint64_t n) {
    std::vector<uint8_t> b(12 + 8 * n, 0);
    std::memcpy(b.data(), &n, 8);
    return b;
}

// A piece of output.bin that does not get to the device: the graph is not
// built over what lies there.  Copies of the caller's own thread go through
// (after one of a helper's has failed).
int graph_input_copy_fails() {
    emp_ctx *c = make_ctx();
    const std::vector<uint8_t> bin = one_record(4 << 20);
    const auto self = std::this_thread::get_id();
    std::atomic<int> failed{0};
    emp_graph *g = nullptr;
    if (emp_graph_build(c, bin.data(), bin.size(), 2, &g) != EMP_OK || fake::graph_builds != 1) return 1;
    emp_graph_destroy(g);
    g = nullptr;
    fake::copy_fails = [&]() {
        if (std::this_thread::get_id() != self) {
            ++failed;
            return true;
        }
        for (int k = 0; k < 5000 && !failed; ++k) std::this_thread::sleep_for(std::chrono::milliseconds(1));
        return false;
    };
    const emp_status st = emp_graph_build(c, bin.data(), bin.size(), 2, &g);
    fake::copy_fails = nullptr;
    if (!failed) return std::thread::hardware_concurrency() > 1 ? 2 : 0;
    return st == EMP_E_CUDA && !g && fake::graph_builds == 1 ? 0 : 3;
}

// A helper thread that cannot be made for want of memory: the copy goes on with those there are.
int thread_allocation_fails() {
    emp::HostStage stage;
    std::vector<uint8_t> in(32 << 20), out(in.size());
    for (size_t i = 0; i < in.size(); i += 4096) in[i] = (uint8_t)(i >> 12);
    for (int n = 1; n <= 12; ++n) {
        std::fill(out.begin(), out.end(), 0);
        alloc_countdown = n;
        const cudaError_t e = stage.to_device(0, out.data(), in.data(), in.size(), nullptr);
        alloc_countdown = 0;
        if (e != cudaSuccess || out != in) return n;
    }
    return 0;
}

// Graphs read, written out and destroyed by other threads than the one that
// uses their context, and beside the context's end (run under a race detector).
int graphs_from_threads() {
    emp_ctx *c = make_ctx();
    const std::vector<uint8_t> bin = one_record(3);
    auto build = [&](uint64_t reads) {
        emp_graph *g = nullptr;
        if (emp_graph_build(c, bin.data(), bin.size(), reads, &g) != EMP_OK) std::abort();
        return g;
    };
    emp_graph *shared = build(2000);
    std::mutex mu;
    std::vector<emp_graph *> made;
    std::atomic<bool> over{false};
    std::atomic<int> wrong{0};
    auto destroyer = [&]() {
        for (;;) {
            const bool last = over;
            emp_graph *g = nullptr;
            {
                std::lock_guard<std::mutex> l(mu);
                if (!made.empty()) {
                    g = made.back();
                    made.pop_back();
                }
            }
            if (g) emp_graph_destroy(g);
            else if (last) return;
        }
    };
    auto reader = [&]() {
        std::vector<uint32_t> order(4000);
        std::vector<uint64_t> starts(4001);
        for (int k = 0; k < 20; ++k) {
            if (emp_graph_write_gfa(shared, "/dev/null", 50) != EMP_OK) ++wrong;
            if (emp_graph_unitigs(shared, order.data(), order.size(), starts.data(), starts.size()) != EMP_OK) ++wrong;
            for (uint32_t u = 0; u < 4000; ++u) wrong += order[u] != u || starts[u] != u;
        }
    };
    std::thread a(destroyer), b(reader), d(reader);
    for (int k = 0; k < 300; ++k) {
        emp_graph *g = build(20);
        std::lock_guard<std::mutex> l(mu);
        made.push_back(g);
    }
    b.join();
    d.join();
    for (int k = 0; k < 300; ++k) {
        emp_graph *g = build(20);
        std::lock_guard<std::mutex> l(mu);
        made.push_back(g);
    }
    emp_ctx_destroy(c);
    over = true;
    a.join();
    emp_graph_destroy(shared);
    return wrong ? 1 : fake::pool_bytes ? 2 : 0;
}

// An open graph's arrays on the device count, and make room for a job: under a
// budget, and on a device that is full.
int graphs_make_room() {
    emp_ctx *c = make_ctx();
    emp_job *j = fed_job(c);
    if (emp_job_run(j, nullptr) != EMP_OK) return 1;
    const long job_bytes = fake::pool_bytes;
    emp_job_destroy(j);
    emp_ctx_destroy(c);
    const std::vector<uint8_t> bin = one_record(3);
    constexpr uint64_t kNodes = 2000000;  // 24 MB on the device
    for (const bool budget : {true, false}) {
        const long limit = job_bytes + (20 << 20);
        c = make_ctx(budget ? (uint64_t)limit : 0);
        emp_graph *g = nullptr, *g2 = nullptr;
        if (emp_graph_build(c, bin.data(), bin.size(), kNodes / 2, &g) != EMP_OK) return 2;
        if (emp_graph_build(c, bin.data(), bin.size(), 10, &g2) != EMP_OK) return 3;
        if (!budget) fake::pool_refuses = [&](size_t n) { return fake::pool_bytes + (long)n > limit; };
        j = fed_job(c);
        const emp_status st = emp_job_run(j, nullptr);
        fake::pool_refuses = nullptr;
        if (st != EMP_OK) return 4;
        if (fake::pool_bytes > limit) return 5;
        emp_job_destroy(j);
        std::vector<uint32_t> order(kNodes);
        std::vector<uint64_t> starts(kNodes + 1);
        for (emp_graph *x : {g, g2}) {
            emp_graph_stats gs;
            emp_graph_get_stats(x, &gs);
            if (emp_graph_unitigs(x, order.data(), kNodes, starts.data(), kNodes + 1) != EMP_OK) return 6;
            for (uint64_t u = 0; u < gs.nodes; ++u)
                if (order[u] != u || starts[u] != u) return 7;
            if (starts[gs.nodes] != gs.nodes) return 8;
            if (emp_graph_write_gfa(x, "/dev/null", 50) != EMP_OK) return 9;
            emp_graph_destroy(x);
        }
        emp_ctx_destroy(c);
        if (fake::pool_bytes) return 10;
    }
    return 0;
}

// A sort whose working set could not grow leaves one that the next, smaller sort can use.
int sort_room_refused() {
    emp_ctx *c = make_ctx();
    std::vector<uint64_t> k(100000);
    std::vector<uint32_t> v(k.size());
    for (int refused = 0; refused < 3; ++refused) {
        if (emp_sort_pairs(c, k.data(), v.data(), 1000 << refused, nullptr) != EMP_OK || !fake::sort_buffers) return 1;
        int asked = 0;
        fake::malloc_refuses = [&](size_t) { return asked++ >= refused; };
        const emp_status st = emp_sort_pairs(c, k.data(), v.data(), k.size(), nullptr);
        fake::malloc_refuses = nullptr;
        if (st != EMP_E_NOMEM) return refused ? 0 : 2;  // 0: the buffers had been grown before
        if (emp_sort_pairs(c, k.data(), v.data(), 500, nullptr) != EMP_OK || !fake::sort_buffers) return 3;
    }
    emp_ctx_destroy(c);
    return 0;
}

// A server step that ends early, at its second launch: the jobs of its first
// launch and those just admitted come back with the status, the long job that
// was to share its rounds stays, and the next step goes on.
int step_ends_early() {
    emp_ctx *c = make_ctx();
    emp_server_params p;
    emp_server_params_default(&p);
    p.share_min_entries = 500;
    emp_server *srv = nullptr;
    if (emp_server_create(c, &p, &srv) != EMP_OK) return 1;
    emp_job *small = fed_job(c), *large = fed_job(c, 40000), *late[2] = {fed_job(c), fed_job(c)};
    emp_job *back[8];
    int n = 0, queued, flying, done;
    emp_server_submit(srv, small);
    emp_server_submit(srv, large);
    if (emp_server_step(srv, back, 8, &n) != EMP_OK || n) return 2;
    for (emp_job *j : late) emp_server_submit(srv, j);
    fake::on_bucket = []() { return cudaErrorUnknown; };
    if (emp_server_step(srv, back, 8, &n) != EMP_E_CUDA || n != 3) return 3;
    fake::on_bucket = nullptr;
    for (int k = 0; k < n; ++k)
        if (back[k] == large || emp_job_status(back[k]) != EMP_E_CUDA) return 4;
    emp_server_counts(srv, &queued, &flying, &done);
    if (queued || flying != 1 || done) return 5;
    if (emp_server_step(srv, back, 8, &n) != EMP_OK || n != 1 || back[0] != large) return 6;
    if (emp_job_status(large) != EMP_OK) return 7;
    emp_job_reset(small);  // and are free for the next set
    if (emp_job_feed_fastq(small, "A", 1, 1) != EMP_OK || emp_job_run(small, nullptr) != EMP_OK) return 8;
    for (emp_job *j : {small, large, late[0], late[1]})
        if (emp_job_destroy(j) != EMP_OK) return 9;
    emp_server_destroy(srv);
    emp_ctx_destroy(c);
    return fake::pool_bytes ? 10 : 0;
}

// Calls on a graph leave the calling thread's device as it is.
int graph_keeps_the_device() {
    emp_ctx *c = make_ctx();
    const std::vector<uint8_t> bin = one_record(3);
    emp_graph *g[3] = {};
    for (emp_graph *&x : g)
        if (emp_graph_build(c, bin.data(), bin.size(), 10, &x) != EMP_OK) return 1;
    std::vector<uint32_t> order(20);
    std::vector<uint64_t> starts(21);
    cudaSetDevice(1);
    if (emp_graph_unitigs(g[0], order.data(), 20, starts.data(), 21) != EMP_OK || fake::device != 1) return 2;
    if (emp_graph_write_gfa(g[1], "/dev/null", 50) != EMP_OK || fake::device != 1) return 3;
    for (emp_graph *x : g)
        if (emp_graph_destroy(x) != EMP_OK || fake::device != 1) return 4;
    emp_ctx_destroy(c);
    return 0;
}

}  // namespace

int main(int argc, char **argv) {
    const std::string name = argc > 1 ? argv[1] : "";
    if (name == "rebuilt_list_times_out") return rebuilt_list_times_out();
    if (name == "graph_input_copy_fails") return graph_input_copy_fails();
    if (name == "thread_allocation_fails") return thread_allocation_fails();
    if (name == "graphs_from_threads") return graphs_from_threads();
    if (name == "graphs_make_room") return graphs_make_room();
    if (name == "sort_room_refused") return sort_room_refused();
    if (name == "step_ends_early") return step_ends_early();
    if (name == "graph_keeps_the_device") return graph_keeps_the_device();
    return 99;
}
