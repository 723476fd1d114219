// select.cu — Filter as a streaming operator, and Project materialised on the
// device.
//
// vexq_filter_open/next/close replace exec.NewFilter over a TableScan
// (exec/filter.go:40-78, exec/scan.go:199-236): the predicate runs once over
// every row group the zone maps keep (one launch, a selection bitmap), then
// every 1024-row block's selection vector is built on the device — per-block
// counts, an exclusive scan, and one warp a block writing its uint16 row
// indices in order — and all of them come back in one copy. next() hands out
// the blocks in row order with the scan's batch (the table's columns, read
// from a pinned host mirror of the HBM columns) and the block's SelVec,
// skipping blocks where no row survives, as Filter.Next does; the views stay
// valid until the next call.
//
// vexq_project_run replaces exec.NewProject over that filter
// (exec/project.go:64-128): the projected expressions are evaluated on the
// device for the kept rows only and written compacted in row order (what
// Project.materialize does with a SelVec), then served in 1024-row batches
// by vexq_result_next.
#include <algorithm>
#include <cstring>

#include "assemble.h"

namespace vq {
cudaStream_t plan_stream(Plan& p);

namespace {

// 32 bits of the bitmap starting at row r (r need not be a multiple of 32; the
// word array carries padding words past the last row)
__device__ __forceinline__ unsigned bits_at(const unsigned* w, long long r) {
    const long long i = r >> 5;
    const int s = (int)(r & 31);
    return s ? (w[i] >> s) | (w[i + 1] << (32 - s)) : w[i];
}

__device__ __forceinline__ unsigned lane_bits(const unsigned* w, long long row0, int len, int lane) {
    const int lo = lane * 32;
    if (lo >= len) return 0u;
    const unsigned b = bits_at(w, row0 + lo);
    const int n = len - lo;
    return n >= 32 ? b : b & ((1u << n) - 1u);
}

// Kept rows of each block (one warp a block).
__global__ void k_block_count(const unsigned* words, const long long* row0, const int* len, int nb, long long* cnt) {
    const int warp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (warp >= nb) return;
    int c = __popc(lane_bits(words, row0[warp], len[warp], lane));
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) cnt[warp] = c;
}

// Each block's SelVec at its offset: lane l writes the kept rows among the
// block's rows 32l..32l+31, after the kept rows of lanes below it.
__global__ void k_block_selvec(const unsigned* words, const long long* row0, const int* len, int nb, const long long* off,
                               unsigned short* sel) {
    const int warp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
    if (warp >= nb) return;
    unsigned b = lane_bits(words, row0[warp], len[warp], lane);
    const int c = __popc(b);
    int inc = c;
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    unsigned short* out = sel + off[warp] + (inc - c);
    while (b) {
        const int i = __ffs(b) - 1;
        *out++ = (unsigned short)(lane * 32 + i);
        b &= b - 1u;
    }
}

// Kept rows of each 128-row chunk (four bitmap words).
__global__ void k_chunk_count(const unsigned* words, long long nck, long long* cnt) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < nck; c += (long long)gridDim.x * blockDim.x) {
        const uint4 w = reinterpret_cast<const uint4*>(words)[c];
        cnt[c] = __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
    }
}

// Exclusive scan of n 64-bit counts in place, in three steps: each 1024-entry
// tile scanned by one block (tile totals out), the totals scanned by one
// block, the totals added back. out[n] receives the grand total.
__device__ __forceinline__ long long block_incl_scan(long long v, long long* sh) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        const long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) sh[warp] = v;
    __syncthreads();
    if (warp == 0) {
        long long s = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += t;
        }
        sh[lane] = s;
    }
    __syncthreads();
    const long long r = v + (warp ? sh[warp - 1] : 0);
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(1024) k_scan64_tiles(long long* a, long long n, long long* tiles) {
    __shared__ long long sh[32];
    const long long i = blockIdx.x * 1024LL + threadIdx.x;
    const long long v = i < n ? a[i] : 0;
    const long long inc = block_incl_scan(v, sh);
    if (i < n) a[i] = inc - v;
    if (threadIdx.x == 1023) tiles[blockIdx.x] = inc;
}

__global__ void __launch_bounds__(1024) k_scan64_totals(long long* tiles, long long nt, long long* total) {
    __shared__ long long sh[32];
    __shared__ long long last;
    long long carry = 0;  // sum of the earlier 1024-entry rounds
    for (long long b = 0; b < nt; b += 1024) {
        const long long i = b + threadIdx.x;
        const long long v = i < nt ? tiles[i] : 0;
        const long long inc = block_incl_scan(v, sh);
        if (i < nt) tiles[i] = carry + inc - v;
        if (threadIdx.x == 1023) last = inc;
        __syncthreads();
        carry += last;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_scan64_add(long long* a, long long n, const long long* tiles) {
    const long long i = blockIdx.x * 1024LL + threadIdx.x;
    if (i < n) a[i] += tiles[blockIdx.x];
}

// Exclusive scan of a[0..n) in place (a needs no padding); *total (device)
// gets the sum. tiles: ceil(n / 1024) entries of scratch.
void scan64(long long* a, long long n, long long* tiles, long long* total, cudaStream_t s) {
    const long long nt = std::max<long long>(1, (n + 1023) / 1024);
    k_scan64_tiles<<<(unsigned)nt, 1024, 0, s>>>(a, n, tiles);
    launch_check(s, "k_scan64_tiles");
    k_scan64_totals<<<1, 1024, 0, s>>>(tiles, nt, total);
    launch_check(s, "k_scan64_totals");
    k_scan64_add<<<(unsigned)nt, 1024, 0, s>>>(a, n, tiles);
    launch_check(s, "k_scan64_add");
    VQ_CUDA(cudaGetLastError());
}

// Projected rows from raw 8-byte images and validity bytes to the result's
// block: each column in its final width with its validity bitmap. One warp an
// item of 32 rows of one column; bound by the block's PCIe writes.
struct ProjectCols {
    int n;
    struct {
        const unsigned long long* v;
        const unsigned char* ok;
        long long vals, valid;
        int width;
    } c[8];
};
__global__ void __launch_bounds__(256) k_project_out(const __grid_constant__ ProjectCols p, long long rows, char* out) {
    const int lane = threadIdx.x & 31;
    const long long items = (rows + 31) / 32 * p.n, nw = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < items; i += nw) {
        const int j = (int)(i % p.n);
        const long long r = i / p.n * 32 + lane;
        const bool in = r < rows;
        const unsigned long long v = in ? p.c[j].v[r] : 0ull;
        const unsigned word = __ballot_sync(0xffffffffu, in && p.c[j].ok[r]);
        if (in) {
            if (p.c[j].width == 8) reinterpret_cast<unsigned long long*>(out + p.c[j].vals)[r] = v;
            else if (p.c[j].width == 4) reinterpret_cast<unsigned*>(out + p.c[j].vals)[r] = (unsigned)v;
            else reinterpret_cast<unsigned char*>(out + p.c[j].vals)[r] = (unsigned char)v;
        }
        if (lane == 0) reinterpret_cast<unsigned*>(out + p.c[j].valid)[r >> 5] = word;
    }
}

int type_width(int t) { return (t == VEXQ_TYPE_INT64 || t == VEXQ_TYPE_FLOAT64) ? 8 : t == VEXQ_TYPE_BOOL ? 1 : 4; }

// The table's columns in pinned host memory, copied from HBM (the columns'
// authoritative copy) on first use and again after the table is re-filled.
struct HostMirror {
    std::vector<std::unique_ptr<PinnedBuf>> vals, valid;
    uint64_t version = ~0ull;
};
std::mutex g_mirror_mu;
std::map<const Table*, std::unique_ptr<HostMirror>> g_mirrors;

}  // namespace

// Plans kept per table: the most recent kKept, each holding at most kKeptBytes
// of device and of pinned memory between calls (larger buffers are freed with
// the call that grew them, and allocated again by the next). A call used to
// compile its plan, create a stream and allocate every buffer: about 450 us of a
// 6M-row selection bitmap's 655. Over all tables at most kAllKept plans and
// kAllBytes of each memory are kept; the least recently used go first, and a
// table's go with it.
struct KeptPlan {
    std::string key;
    std::unique_ptr<Plan> p;
    size_t dev = 0, pinned = 0;  // bytes it holds
    uint64_t used = 0;
};
struct SelectPlans {
    std::vector<KeptPlan> kept;
    SelectPlans();
    ~SelectPlans();
};
namespace {
constexpr size_t kKept = 8, kKeptBytes = 32u << 20, kAllKept = 64, kAllBytes = 128u << 20;
// every table's plans, and what they hold together (guarded by mu)
struct AllKept {
    std::mutex mu;
    std::vector<SelectPlans*> tables;
    size_t n = 0, dev = 0, pinned = 0;
    uint64_t clock = 0;
    KeptPlan take(SelectPlans& s, size_t i) {
        KeptPlan k = std::move(s.kept[i]);
        s.kept.erase(s.kept.begin() + i);
        n--;
        dev -= k.dev;
        pinned -= k.pinned;
        return k;
    }
    // the least recently used plan of one table, or of all (null)
    KeptPlan oldest(SelectPlans* of) {
        SelectPlans* at = nullptr;
        size_t ix = 0;
        for (SelectPlans* s : tables)
            if (!of || s == of)
                for (size_t i = 0; i < s->kept.size(); i++)
                    if (!at || s->kept[i].used < at->kept[ix].used) {
                        at = s;
                        ix = i;
                    }
        return take(*at, ix);
    }
};
AllKept& all_kept() {
    static auto* a = new AllKept;  // (tables may outlive the statics)
    return *a;
}
}  // namespace

SelectPlans::SelectPlans() { all_kept().tables.push_back(this); }
SelectPlans::~SelectPlans() {
    AllKept& a = all_kept();
    std::vector<KeptPlan> gone;  // plans are destroyed without the lock
    std::lock_guard<std::mutex> lk(a.mu);
    while (!kept.empty()) gone.push_back(a.take(*this, kept.size() - 1));
    a.tables.erase(std::find(a.tables.begin(), a.tables.end(), this));
}

SelectLease::SelectLease(Table& tb, char kind, const vexq_expr* nodes, int nnodes, const int32_t* children, int nchildren, int pred,
                         const int32_t* roots, int nroots)
    : t(tb) {
    // the expression, whole: a plan is reused only for the same one
    auto raw = [&](const void* q, size_t n) { key.append((const char*)q, n); };
    key.push_back(kind);
    raw(&pred, sizeof pred);
    raw(&nroots, sizeof nroots);
    if (nroots > 0 && roots) raw(roots, (size_t)nroots * 4);
    raw(&nchildren, sizeof nchildren);
    if (nchildren > 0 && children) raw(children, (size_t)nchildren * 4);
    for (int i = 0; i < nnodes; i++) {
        const vexq_expr& e = nodes[i];
        const int32_t head[6] = {e.kind, e.op, e.column, e.lit_kind, e.child0, e.nchildren};
        raw(head, sizeof head);
        raw(&e.lit_int, 8);
        raw(&e.lit_float, 8);
        // (lit_str of any other node is the caller's to leave unset)
        const char* s = e.kind == VEXQ_E_LITERAL && e.lit_kind == VEXQ_LIT_STRING ? e.lit_str : nullptr;
        const int64_t len = s ? (int64_t)std::strlen(s) : -1;
        raw(&len, 8);
        if (len > 0) raw(s, (size_t)len);
    }
    {
        AllKept& a = all_kept();
        std::vector<KeptPlan> gone;
        std::lock_guard<std::mutex> lk(a.mu);
        if (!t.selects) t.selects = std::make_shared<SelectPlans>();
        std::vector<KeptPlan>& kept = t.selects->kept;
        for (size_t i = kept.size(); i-- > 0;) {
            // a refill that widened a column's range changes what is generated
            if (kept[i].p->range_epoch != t.range_epoch) gone.push_back(a.take(*t.selects, i));
            else if (!p && kept[i].key == key) p = a.take(*t.selects, i).p;
        }
    }
    if (!p) p.reset(kind == 'f' ? compile_filter(&t, nodes, nnodes, children, nchildren, pred)
                                : compile_select(&t, nodes, nnodes, children, nchildren, pred, roots, nroots));
}

void SelectLease::done() {
    DevBuf* bufs[] = {&p->scratch_a, &p->scratch_b, &p->scratch_c, &p->scratch_d};
    KeptPlan k;
    for (DevBuf* b : bufs) k.dev += b->n;
    if (k.dev > kKeptBytes) {
        for (DevBuf* b : bufs) b->release();
        k.dev = 0;
    }
    if (p->h_stage.n > kKeptBytes) p->h_stage.release();
    p->out_pool.trim(kKeptBytes / 2);
    k.dev += p->d_seg.n + p->d_sets.n + p->d_present.n;
    k.pinned = p->h_stage.n + p->out_pool.bytes();
    k.key = std::move(key);
    k.p = std::move(p);
    AllKept& a = all_kept();
    std::vector<KeptPlan> gone;
    std::lock_guard<std::mutex> lk(a.mu);
    SelectPlans& s = *t.selects;
    if (s.kept.size() >= kKept) gone.push_back(a.oldest(&s));
    k.used = ++a.clock;
    a.n++;
    a.dev += k.dev;
    a.pinned += k.pinned;
    s.kept.push_back(std::move(k));
    while (a.n > kAllKept || a.dev > kAllBytes || a.pinned > kAllBytes) gone.push_back(a.oldest(nullptr));
}

void drop_host_mirror(const Table* t) {
    std::lock_guard<std::mutex> lk(g_mirror_mu);
    g_mirrors.erase(t);
}

namespace {

HostMirror& host_mirror(Table& t, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(g_mirror_mu);
    auto& m = g_mirrors[&t];
    if (!m) m.reset(new HostMirror);
    if (m->version == t.zone_version) return *m;
    m->vals.clear();
    m->valid.clear();
    for (const Column& c : t.cols) {
        auto v = std::make_unique<PinnedBuf>();
        auto b = std::make_unique<PinnedBuf>();
        const size_t nb = (size_t)std::max<int64_t>(t.nrows, 1) * type_width(c.type);
        v->ensure(nb);
        if (t.nrows > 0) VQ_CUDA(cudaMemcpyAsync(v->p, c.values.p, (size_t)t.nrows * type_width(c.type), cudaMemcpyDeviceToHost, s));
        const size_t vb = (size_t)(t.nrows + 7) / 8 + 8;
        b->ensure(vb);
        if (c.nullable && t.nrows > 0) {
            VQ_CUDA(cudaMemcpyAsync(b->p, c.validity.p, (size_t)(t.nrows + 7) / 8, cudaMemcpyDeviceToHost, s));
        } else {
            std::memset(b->p, 0xFF, vb);
        }
        m->vals.push_back(std::move(v));
        m->valid.push_back(std::move(b));
    }
    VQ_CUDA(cudaStreamSynchronize(s));
    m->version = t.zone_version;
    return *m;
}

// Row ranges kept by the zone maps, as the scan's segment list.
ScanSegs kept_segments(const Plan& p, const Table& t, int rgs, int rge) {
    std::vector<uint8_t> m = p.zn_pred >= 0 ? prune_mask(p, t, p.zn_pred, rgs, rge) : std::vector<uint8_t>(t.n_rg, 0);
    if (p.zn_pred < 0)
        for (int rg = rgs; rg < rge; rg++) m[rg] = 1;
    return make_segments(t, m, rgs, rge, 128);
}

// Scan parameters of a select plan over its table.
VQParams select_params(Plan& p, const Table& t, const DevBuf& seg, const ScanSegs& ss) {
    VQParams P;
    std::memset(&P, 0, sizeof P);
    set_plan_constants(p, P);
    set_columns(P, t, false);
    P.seg = seg.as<long long>();
    P.nseg = (int)ss.seg.size() / 3;
    set_one_seg(P, ss.seg);
    P.nchunks = ss.nchunks;
    P.rg_rows = t.rg_rows;
    P.n_rg = t.n_rg;
    P.present = p.d_present.as<unsigned char>();
    for (size_t i = 0, o = 0; i < p.sets.size(); i++) {
        P.sets[i] = p.d_sets.as<unsigned>() + o;
        o += p.sets[i].size();
    }
    return P;
}

void check_range_args(const Table& t, int& rgs, int& rge) {
    if (rge < 0 || rge > t.n_rg) rge = t.n_rg;
    if (rgs < 0 || rgs > rge) fail(VEXQ_EINVAL, "row-group range out of bounds");
}

}  // namespace
}  // namespace vq

using namespace vq;

struct vexq_filter_s {
    std::unique_ptr<Plan> plan;
    Table* t = nullptr;
    HostMirror* mirror = nullptr;
    std::vector<long long> row0;    // per block: first table row
    std::vector<int> len, rg;       // rows and row group
    std::vector<long long> cnt, off;
    PinnedBuf h_sel;                // every block's SelVec, compacted
    long long selected = 0;
    size_t next_block = 0;
    // views of the current batch
    std::vector<vexq_vector_view> views;
    std::vector<std::vector<uint8_t>> vbits;
    std::vector<std::vector<uint32_t>> doff;
    std::vector<std::string> dbytes;
    double kernel_ms = 0;
};

namespace {

template <class F>
int32_t guard_s(F&& f) {
    try {
        set_error("");
        return f();
    } catch (const Status& s) {
        set_error(s.what());
        return s.code;
    } catch (const std::bad_alloc&) {
        set_error("host allocation failed");
        return VEXQ_ENOMEM;
    } catch (const std::exception& e) {
        set_error(e.what());
        return VEXQ_EINVAL;
    }
}

float ev_ms(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0;
    VQ_CUDA(cudaEventElapsedTime(&ms, a, b));
    return ms;
}

struct Events {
    cudaEvent_t a = nullptr, b = nullptr;
    Events() {
        VQ_CUDA(cudaEventCreate(&a));
        VQ_CUDA(cudaEventCreate(&b));
    }
    ~Events() {
        if (a) cudaEventDestroy(a);
        if (b) cudaEventDestroy(b);
    }
};

// The bitmap of the kept rows of segments ss (vq_pmark); words is sized to
// (nrows + kPadRows) / 32 + 8 words and zeroed on stream s first.
void mark_rows(Plan& p, const Table& t, const ScanSegs& ss, DevBuf& words, DevBuf& seg, cudaStream_t s) {
    words.ensure(((size_t)(t.nrows + kPadRows) / 32 + 8) * 4);
    VQ_CUDA(cudaMemsetAsync(words.p, 0, words.n, s));
    if (ss.seg.size() != 3) {  // one range travels in the parameter block
        seg.ensure(std::max<size_t>(ss.seg.size(), 3) * 8);
        h2d(seg.p, ss.seg.data(), ss.seg.size() * 8, s);
    }
    if (ss.nchunks <= 0) return;
    VQParams P = select_params(p, t, seg, ss);
    P.acc_i = words.as<long long>();
    jit_launch(p.k_main, grid_for(p.k_main, ss.nchunks, false, 0), &P, sizeof P, s);
    launch_check(s, "vq_pmark");
}

}  // namespace

extern "C" {

int32_t vexq_filter_open(vexq_table_t table, const vexq_expr* nodes, int32_t nnodes, const int32_t* children,
                         int32_t nchildren, int32_t predicate, int32_t rg_start, int32_t rg_end, vexq_filter_t* out) {
    return guard_s([&]() -> int32_t {
        if (!table || !out || !nodes) fail(VEXQ_EINVAL, "null argument");
        *out = nullptr;
        Table& t = *table->t;
        int rgs = rg_start, rge = rg_end;
        check_range_args(t, rgs, rge);
        std::unique_ptr<vexq_filter_s> f(new vexq_filter_s);
        f->t = &t;
        f->plan.reset(compile_select(&t, nodes, nnodes, children, nchildren, predicate, nullptr, 0));
        Plan& p = *f->plan;
        cudaStream_t s = plan_stream(p);
        f->mirror = &host_mirror(t, s);
        const ScanSegs ss = kept_segments(p, t, rgs, rge);
        // 1024-row blocks of the kept row groups (a block never spans two)
        for (int rg = rgs; rg < rge; rg++) {
            bool kept = false;
            for (size_t i = 0; i + 2 < ss.seg.size(); i += 3)
                if (ss.seg[i] <= t.rg_start(rg) && t.rg_start(rg) < ss.seg[i + 1]) kept = true;
            if (!kept) continue;
            for (int64_t r = t.rg_start(rg); r < t.rg_end(rg); r += VEXQ_BLOCK_ROWS) {
                f->row0.push_back(r);
                f->len.push_back((int)std::min<int64_t>(VEXQ_BLOCK_ROWS, t.rg_end(rg) - r));
                f->rg.push_back(rg);
            }
        }
        const int nb = (int)f->row0.size();
        f->cnt.assign(nb, 0);
        f->off.assign(nb, 0);
        if (nb > 0) {
            Events e;
            DevBuf words, seg, d_row0(nb * 8), d_len(nb * 4), d_cnt((size_t)(nb + 1) * 8),
                d_tiles((size_t)((nb + 1023) / 1024 + 1) * 8), d_total(8), d_sel((size_t)t.nrows * 2 + 16);
            VQ_CUDA(cudaEventRecord(e.a, s));
            mark_rows(p, t, ss, words, seg, s);
            h2d(d_row0.p, f->row0.data(), nb * 8, s);
            h2d(d_len.p, f->len.data(), nb * 4, s);
            const int wb = 256, grid = (int)(((long long)nb * 32 + wb - 1) / wb);
            k_block_count<<<grid, wb, 0, s>>>(words.as<unsigned>(), d_row0.as<long long>(), d_len.as<int>(), nb,
                                              d_cnt.as<long long>());
            launch_check(s, "k_block_count");
            VQ_CUDA(cudaMemcpyAsync(f->cnt.data(), d_cnt.p, nb * 8, cudaMemcpyDeviceToHost, s));
            scan64(d_cnt.as<long long>(), nb, d_tiles.as<long long>(), d_total.as<long long>(), s);
            k_block_selvec<<<grid, wb, 0, s>>>(words.as<unsigned>(), d_row0.as<long long>(), d_len.as<int>(), nb,
                                               d_cnt.as<long long>(), d_sel.as<unsigned short>());
            launch_check(s, "k_block_selvec");
            VQ_CUDA(cudaGetLastError());
            VQ_CUDA(cudaMemcpyAsync(f->off.data(), d_cnt.p, nb * 8, cudaMemcpyDeviceToHost, s));
            VQ_CUDA(cudaMemcpyAsync(&f->selected, d_total.p, 8, cudaMemcpyDeviceToHost, s));
            VQ_CUDA(cudaStreamSynchronize(s));
            f->h_sel.ensure((size_t)std::max<long long>(f->selected, 1) * 2);
            if (f->selected > 0)
                VQ_CUDA(cudaMemcpyAsync(f->h_sel.p, d_sel.p, (size_t)f->selected * 2, cudaMemcpyDeviceToHost, s));
            VQ_CUDA(cudaEventRecord(e.b, s));
            VQ_CUDA(cudaStreamSynchronize(s));
            f->kernel_ms = ev_ms(e.a, e.b);
        }
        // each STRING column's global dictionary, flattened once for the views
        const size_t nc = t.cols.size();
        f->views.assign(nc, vexq_vector_view{});
        f->vbits.assign(nc, std::vector<uint8_t>(VEXQ_BLOCK_ROWS / 8 + 1, 0));
        f->doff.assign(nc, {});
        f->dbytes.assign(nc, {});
        for (size_t c = 0; c < nc; c++) {
            const Column& col = t.cols[c];
            vexq_vector_view& v = f->views[c];
            v.name = col.name.c_str();
            v.type = col.type;
            if (col.type == VEXQ_TYPE_STRING) {
                f->doff[c].push_back(0);
                for (const std::string& k : col.dict.keys) {
                    f->dbytes[c] += k;
                    f->doff[c].push_back((uint32_t)f->dbytes[c].size());
                }
                v.dict_str_off = f->doff[c].data();
                v.dict_bytes = f->dbytes[c].data();
                v.dict_len = (int32_t)col.dict.keys.size();
            }
        }
        *out = f.release();
        return VEXQ_OK;
    });
}

int32_t vexq_filter_next(vexq_filter_t f, vexq_filter_batch* out) {
    return guard_s([&]() -> int32_t {
        if (!f || !out) fail(VEXQ_EINVAL, "null argument");
        std::memset(out, 0, sizeof *out);
        while (f->next_block < f->row0.size() && f->cnt[f->next_block] == 0) f->next_block++;
        if (f->next_block >= f->row0.size()) return VEXQ_OK;  // EOF: length 0
        const size_t b = f->next_block++;
        const Table& t = *f->t;
        const long long r0 = f->row0[b];
        const int n = f->len[b];
        for (size_t c = 0; c < t.cols.size(); c++) {
            vexq_vector_view& v = f->views[c];
            v.values = (const char*)f->mirror->vals[c]->p + (size_t)r0 * type_width(t.cols[c].type);
            // the block's validity bits from bit 0 (the mirror's bitmap is
            // table-wide; a block need not start on a byte)
            const uint8_t* src = (const uint8_t*)f->mirror->valid[c]->p;
            std::vector<uint8_t>& dst = f->vbits[c];
            std::fill(dst.begin(), dst.end(), 0);
            const int sh = (int)(r0 & 7);
            const long long b0 = r0 >> 3;
            for (int i = 0; i < (n + 7) / 8; i++) {
                unsigned x = (unsigned)src[b0 + i] >> sh;
                if (sh) x |= (unsigned)src[b0 + i + 1] << (8 - sh);
                dst[i] = (uint8_t)x;
            }
            if (n & 7) dst[(n - 1) / 8] &= (uint8_t)((1u << (n & 7)) - 1u);
            v.validity = dst.data();
        }
        out->ncols = (int32_t)t.cols.size();
        out->length = (int32_t)f->cnt[b];
        out->physical = n;
        out->rg = f->rg[b];
        out->row0 = r0;
        out->sel = (const uint16_t*)f->h_sel.p + f->off[b];
        out->cols = f->views.data();
        return VEXQ_OK;
    });
}

int32_t vexq_filter_stats(vexq_filter_t f, int64_t* selected, int64_t* blocks, double* kernel_ms) {
    return guard_s([&]() -> int32_t {
        if (!f) fail(VEXQ_EINVAL, "null argument");
        if (selected) *selected = f->selected;
        if (blocks) *blocks = (int64_t)f->row0.size();
        if (kernel_ms) *kernel_ms = f->kernel_ms;
        return VEXQ_OK;
    });
}

int32_t vexq_filter_close(vexq_filter_t f) {
    delete f;
    return VEXQ_OK;
}

int32_t vexq_project_run(vexq_table_t table, const vexq_expr* nodes, int32_t nnodes, const int32_t* children,
                         int32_t nchildren, int32_t predicate, const int32_t* roots, const char* const* names,
                         int32_t nexprs, int32_t rg_start, int32_t rg_end, vexq_result_t* out) {
    return guard_s([&]() -> int32_t {
        if (!table || !out || !nodes || !roots || nexprs <= 0) fail(VEXQ_EINVAL, "null argument or no expressions");
        *out = nullptr;
        Table& t = *table->t;
        int rgs = rg_start, rge = rg_end;
        check_range_args(t, rgs, rge);
        SelectLease lease(t, 'p', nodes, nnodes, children, nchildren, predicate, roots, nexprs);
        Plan& p = *lease.p;
        cudaStream_t s = plan_stream(p);
        const ScanSegs ss = kept_segments(p, t, rgs, rge);
        std::unique_ptr<vexq_result_s> r(new vexq_result_s);
        r->cols.resize(nexprs);
        for (int j = 0; j < nexprs; j++) {
            const INode& n = p.ir[p.key_nodes[j]];
            OutColumn& oc = r->cols[j];
            oc.name = names && names[j] ? names[j] : ("col" + std::to_string(j));
            oc.type = n.type;
            if (n.type == VEXQ_TYPE_STRING) oc.dict = &t.cols[n.col].dict;
        }
        long long total = 0;
        ensure_events(p);
        VQ_CUDA(cudaEventRecord(p.ev[0], s));
        int launches = 0;
        bool direct = false;  // columns written by the device into the result's block
        if (ss.nchunks > 0) {
            DevBuf &words = p.scratch_a, &seg = p.d_seg, &scr = p.scratch_b;
            mark_rows(p, t, ss, words, seg, s);
            const long long nck = (t.nrows + 127) / 128 + 1;
            // chunk offsets | tile totals | grand total
            const size_t b_off = (size_t)(nck + 1) * 8, b_tiles = (size_t)((nck + 1023) / 1024 + 1) * 8;
            scr.ensure(b_off + b_tiles + 8);
            long long* d_off = scr.as<long long>();
            long long* d_tiles = (long long*)(scr.as<char>() + b_off);
            long long* d_total = (long long*)(scr.as<char>() + b_off + b_tiles);
            const int cg = (int)std::min<long long>((nck + 255) / 256, (long long)sm_count() * 8);
            k_chunk_count<<<cg, 256, 0, s>>>(words.as<unsigned>(), nck, d_off);
            launch_check(s, "k_chunk_count");
            scan64(d_off, nck, d_tiles, d_total, s);
            p.h_stage.ensure(8);
            VQ_CUDA(cudaMemcpyAsync(p.h_stage.p, d_total, 8, cudaMemcpyDeviceToHost, s));
            VQ_CUDA(cudaStreamSynchronize(s));
            total = *(const long long*)p.h_stage.p;
            launches = 5;
            if (total > 0) {
                const int ng = (nexprs + 7) / 8, nb = std::min(nexprs, 8);
                // eight expressions' images and validity bytes at a time
                const size_t b_v = ((size_t)total * 8 + 255) & ~(size_t)255, b_m = ((size_t)total + 255) & ~(size_t)255;
                p.scratch_c.ensure((b_v + b_m) * nb);
                char* dv = p.scratch_c.as<char>();
                char* dm = dv + b_v * nb;
                VQParams P = select_params(p, t, seg, ss);
                P.acc_i = words.as<long long>();
                P.first = d_off;
                for (int j = 0; j < nb; j++) {
                    P.qpay[j] = (unsigned long long*)(dv + b_v * j);
                    P.qpayv[j] = (unsigned char*)(dm + b_m * j);
                }
                // the result's block: every column's values and bitmap. Up to
                // 64 MB pinned (larger results come back column by column)
                std::vector<std::pair<size_t, size_t>> at(nexprs);
                size_t bytes = 0;
                for (int j = 0; j < nexprs; j++) {
                    at[j].first = bytes;
                    bytes += ((size_t)total * type_width(r->cols[j].type) + 127) & ~(size_t)127;
                    at[j].second = bytes;
                    bytes += ((size_t)(total + 31) / 32 * 4 + 127) & ~(size_t)127;
                }
                bool lend = true;
                std::shared_ptr<OutBlock> blk;
                if (bytes <= (64u << 20)) blk = p.out_pool.acquire(bytes, lend);
                direct = blk != nullptr;
                if (!direct)
                    for (auto& oc : r->cols) {
                        oc.v.resize(total);
                        oc.valid.resize(total);
                    }
                for (int g = 0; g < ng; g++) {
                    P.mode = g;
                    jit_launch(p.k_build, grid_for(p.k_build, ss.nchunks, false, 0), &P, sizeof P, s);
                    launch_check(s, "vq_pwrite");
                    launches++;
                    const int j0 = g * 8, j1 = std::min(nexprs, g * 8 + 8);
                    if (direct) {
                        ProjectCols pc;
                        std::memset(&pc, 0, sizeof pc);
                        pc.n = j1 - j0;
                        for (int j = j0; j < j1; j++)
                            pc.c[j - j0] = {P.qpay[j - j0], P.qpayv[j - j0], (long long)at[j].first, (long long)at[j].second,
                                            type_width(r->cols[j].type)};
                        k_project_out<<<2 * sm_count(), 256, 0, s>>>(pc, total, blk->dev);
                        VQ_CUDA(cudaGetLastError());
                        launch_check(s, "k_project_out");
                        launches++;
                        continue;
                    }
                    for (int j = j0; j < j1; j++) {
                        VQ_CUDA(cudaMemcpyAsync(r->cols[j].v.data(), P.qpay[j % 8], (size_t)total * 8, cudaMemcpyDeviceToHost, s));
                        VQ_CUDA(cudaMemcpyAsync(r->cols[j].valid.data(), P.qpayv[j % 8], (size_t)total, cudaMemcpyDeviceToHost, s));
                    }
                    VQ_CUDA(cudaStreamSynchronize(s));
                }
                if (direct) {
                    VQ_CUDA(cudaEventRecord(p.ev[2], s));
                    VQ_CUDA(cudaStreamSynchronize(s));
                    const char* data = (const char*)blk->pin.p;
                    if (!lend) {  // the pool's blocks are with earlier results: a copy of its own
                        auto own = std::make_shared<OutBlock>();
                        own->heap.reset(new char[bytes]);
                        std::memcpy(own->heap.get(), data, bytes);
                        data = own->heap.get();
                        blk = own;
                    }
                    r->block = blk;
                    for (int j = 0; j < nexprs; j++) {
                        OutColumn& oc = r->cols[j];
                        oc.dv = data + at[j].first;
                        oc.dm = (const uint8_t*)data + at[j].second;
                        if (oc.type == VEXQ_TYPE_STRING) oc.flat = flat_dict(t.cols[p.ir[p.key_nodes[j]].col]);
                        oc.dict = nullptr;
                    }
                }
            }
        }
        if (!direct) {
            VQ_CUDA(cudaEventRecord(p.ev[2], s));
            VQ_CUDA(cudaStreamSynchronize(s));
        }
        r->nrows = total;
        own_dictionaries(r.get());
        r->kernel_ms = ev_ms(p.ev[0], p.ev[2]);
        r->scan_ms = r->kernel_ms;
        r->launches = launches;
        r->rows_scanned = ss.rows;
        lease.done();
        *out = r.release();
        return VEXQ_OK;
    });
}

}  // extern "C"
