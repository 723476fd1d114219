// assemble.cu — result columns of a group table written on the device.
//
// The reference hands a HashAggregate's groups out in insertion order
// (exec/aggregate.go:209-216) as typed vectors with validity bitmaps
// (buildOutputBatch, exec/aggregate.go:780-876). k_assemble does that where
// the group table lies: it orders the occupied slots by their first row,
// decodes the keys, finishes the aggregates and writes the columns, in output
// order and final width, straight into a pinned host block that
// vexq_result_next then views without another pass.
//
// Ordering: a group's first row belongs to no other group, so one bit per
// scanned row marks the first rows and a group's output position is the number
// of set bits below its own — a mark, a prefix count and a lookup instead of a
// sort. NULL-keyed groups of the reference's integer-key path come first
// (exec/agg_intkey.go:249-255): they take a bit range ahead of the others'.
//
// One cluster of eight CTAs per table, so the steps (mark, count, place, write)
// are separated by the hardware cluster barrier instead of
// launches, and a batch assembles every table in one launch.
#include <algorithm>
#include <cstring>

#include "assemble.h"
#include "device_common.cuh"

namespace vq {

namespace {

constexpr int kAsmCtas = 8;       // cluster size (portable limit)
constexpr int kAsmThreads = 1024;
constexpr int kRuns = 4;
static_assert(kAsmThreads == 32 * 32 && kRuns <= 32, "one warp adds up a run's 32 warps");
constexpr int kAsmMaxCols = 48;
constexpr long long kOrderMask = (1LL << 56) - 1;  // row part of an order key (bit 56: the phase)

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ long long order_bit(const VQAsmDesc& d, long long f) {
    return (f & kOrderMask) - d.row0 + ((f >> 56) ? d.phase_bits : 0);
}

// One output value: its raw image and whether it is valid.
__device__ __forceinline__ bool asm_value(const VQAsmDesc& d, const VQAsmCol& c, long long slot, unsigned long long& v) {
    v = 0ull;
    if (c.src == ASM_DENSE_KEY) {
        const unsigned long long code = ((unsigned long long)slot / c.stride) % c.domain;
        if (c.nullable && code == c.domain - 1) return false;
        v = code + (unsigned long long)c.vmin;
        return true;
    }
    if (c.src == ASM_PACKED_KEY) {
        const unsigned long long key = slot == d.nslots - 1 ? VQ_EMPTY_KEY : d.keys[slot * d.kst];
        const unsigned long long raw = (key >> c.shift) & (c.bits >= 64 ? ~0ull : ((1ull << c.bits) - 1));
        if (c.domain) {
            if (c.nullable && raw == c.domain - 1) return false;
            v = raw + (unsigned long long)c.vmin;
            return true;
        }
        if (c.date33 && ((raw >> 32) & 1)) return false;
        v = raw;
        return true;
    }
    long long nn = 1;
    if (c.nn >= 0) {
        nn = d.acc_i[(long long)c.nn * d.nslots + slot];
        if (nn == 0) return false;
    }
    if (c.src == ASM_INT) {
        v = (unsigned long long)d.acc_i[(long long)c.slot * d.nslots + slot];
        if (c.width == 1) v = v != 0;
    } else if (c.src == ASM_FKEY) {
        v = (unsigned long long)__double_as_longlong(vq_fkey_inv((unsigned long long)d.acc_i[(long long)c.slot * d.nslots + slot]));
    } else {
        const long long at = (long long)c.slot * d.nslots + slot;
        double x = vq_fx_result(d.acc_fx + at * 4, d.fx_lsb[c.slot], d.special[at]);
        if (c.src == ASM_AVG) x = x / (double)nn;
        v = (unsigned long long)__double_as_longlong(x);
    }
    return true;
}

// Output rows [32 * (item / ncols), …) of column item % ncols, one warp an
// item: stores over PCIe are whole lines and the ballot is the validity word.
__device__ __forceinline__ void asm_write(const VQAsmDesc& d, const VQAsmCol* cols, char* out, long long rows, long long warp0,
                                          long long nwarps) {
    const int lane = threadIdx.x & 31;
    const long long items = (rows + 31) / 32 * d.ncols;
    for (long long item = warp0; item < items; item += nwarps) {
        const long long r = (item / d.ncols) * 32 + lane;
        const VQAsmCol& c = cols[item % d.ncols];
        unsigned long long v = 0ull;
        const bool ok = r < rows && asm_value(d, c, (long long)__ldcg(d.perm + r), v);
        const unsigned word = __ballot_sync(0xffffffffu, ok);
        if (r < rows) {
            if (c.width == 8) reinterpret_cast<unsigned long long*>(out + c.vals)[r] = v;
            else if (c.width == 4) reinterpret_cast<unsigned*>(out + c.vals)[r] = (unsigned)v;
            else reinterpret_cast<unsigned char*>(out + c.vals)[r] = (unsigned char)v;
        }
        if (lane == 0) reinterpret_cast<unsigned*>(out + c.valid)[r >> 5] = word;
    }
}

// The run's stamps and this moment, to the host.
__device__ void asm_clock(const VQAsmDesc& d, VQAsmHdr* h) {
    for (int i = 0; i < VQ_CLK_END; i++) h->clk[i] = __ldcg(d.clk + i);
    h->clk[VQ_CLK_END] = vq_clock();
}

// Bound by latency, not bytes: 1,000 groups of a 4M-row scan read 500 KB of
// marks and 68 KB of table. The first-row bitmap is divided over the CTAs for
// the count, slots and output rows over all of the cluster's threads.
__global__ void __cluster_dims__(kAsmCtas, 1, 1) __launch_bounds__(kAsmThreads)
k_assemble(const VQAsmDesc* descs, char* base, char* const* basep) {
    __shared__ VQAsmDesc d;
    __shared__ VQAsmCol cols[kAsmMaxCols];
    __shared__ unsigned warp_sum[kRuns][kAsmThreads / 32], run_sum[kRuns];
    __shared__ unsigned cta_base[kAsmCtas + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)(blockIdx.x % kAsmCtas);
    {
        const VQAsmDesc* g = descs + blockIdx.x / kAsmCtas;
        static_assert(sizeof(VQAsmDesc) % 4 == 0 && sizeof(VQAsmCol) % 4 == 0, "copied by words");
        for (int i = tid; i < (int)(sizeof d / 4); i += kAsmThreads) ((int*)&d)[i] = ((const int*)g)[i];
        __syncthreads();
        for (int i = tid; i < d.ncols * (int)(sizeof(VQAsmCol) / 4); i += kAsmThreads) ((int*)cols)[i] = ((const int*)d.cols)[i];
    }
    char* out = (basep ? *basep : base) + d.out;
    const int gtid = rank * kAsmThreads + tid;
    constexpr int kAll = kAsmCtas * kAsmThreads;
    // words [w0, w1) of the bitmap are this CTA's
    const int per = (((int)d.nwords + kAsmCtas - 1) / kAsmCtas + 3) & ~3;
    const int w0 = min((int)d.nwords, rank * per), w1 = min((int)d.nwords, w0 + per);
    // the bitmap is clear: the last run left it so
    long long mine = -1;  // the first-row bit of the thread's first slot
    for (long long i = gtid; i < d.nslots; i += kAll) {
        const long long cnt = d.acc_i[i], f = d.first[i * d.kst];
        if (cnt == 0) continue;  // slot 0 of the integer bank is the row count
        const long long b = order_bit(d, f);
        atomicOr(d.bits + (b >> 5), 1u << (b & 31));
        if (i == gtid) mine = b;
    }
    cluster_sync();
    // set bits before each group of four words: a round takes kRuns runs of
    // 4,096 words, a thread one uint4 of each, and one warp a run adds up the
    // run's warps
    unsigned carry = 0u;
    for (int b = w0; b < w1; b += kAsmThreads * 4 * kRuns) {
        unsigned sum[kRuns], incl[kRuns];
#pragma unroll
        for (int k = 0; k < kRuns; k++) {
            const int i = b + (k * kAsmThreads + tid) * 4;
            const uint4 v = i < w1 ? __ldcg(reinterpret_cast<const uint4*>(d.bits + i)) : make_uint4(0u, 0u, 0u, 0u);
            incl[k] = sum[k] = __popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w);
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
#pragma unroll
            for (int k = 0; k < kRuns; k++) {
                const unsigned t = __shfl_up_sync(0xffffffffu, incl[k], o);
                if (lane >= o) incl[k] += t;
            }
        if (lane == 31)
#pragma unroll
            for (int k = 0; k < kRuns; k++) warp_sum[k][warp] = incl[k];
        __syncthreads();
        if (warp < kRuns) {
            const unsigned own = warp_sum[warp][lane];
            unsigned t = own;
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned u = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += u;
            }
            warp_sum[warp][lane] = t - own;
            if (lane == 31) run_sum[warp] = t;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kRuns; k++) {
            const int i = b + (k * kAsmThreads + tid) * 4;
            if (i < w1) d.pref[i >> 2] = carry + warp_sum[k][warp] + incl[k] - sum[k];
            carry += run_sum[k];
        }
        __syncthreads();
    }
    if (tid == 0) d.pref[d.nwords / 4 + rank] = carry;
    cluster_sync();
    if (warp == 0) {
        const unsigned own = lane < kAsmCtas ? __ldcg(d.pref + d.nwords / 4 + lane) : 0u;
        unsigned incl = own;
        for (int o = 1; o <= kAsmCtas; o <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += t;
        }
        if (lane <= kAsmCtas) cta_base[lane] = incl - own;
    }
    __syncthreads();
    const long long n = cta_base[kAsmCtas];
    for (long long i = gtid; i < d.nslots; i += kAll) {
        long long b = mine;
        if (i != gtid) b = d.acc_i[i] != 0 ? order_bit(d, d.first[i * d.kst]) : -1;
        if (b < 0) continue;
        const int w = (int)(b >> 5);
        const uint4 q = __ldcg(reinterpret_cast<const uint4*>(d.bits + (w & ~3)));
        const unsigned below = (1u << (b & 31)) - 1u;
        const int at = w & 3;  // words of the four before the group's, and its bits below
        const long long pos = (long long)cta_base[w / per] + __ldcg(d.pref + (w >> 2)) +
                              __popc(at > 0 ? q.x : q.x & below) + __popc(at > 1 ? q.y : at == 1 ? q.y & below : 0u) +
                              __popc(at > 2 ? q.z : at == 2 ? q.z & below : 0u) + __popc(at == 3 ? q.w & below : 0u);
        if (pos < d.cap_rows) d.perm[pos] = (unsigned)i;
    }
    cluster_sync();
    for (int w = w0 + tid * 4; w < w1; w += kAsmThreads * 4) *reinterpret_cast<uint4*>(d.bits + w) = make_uint4(0u, 0u, 0u, 0u);
    if (d.write) asm_write(d, cols, out, min(n, d.cap_rows), gtid >> 5, kAll / 32);
    if (gtid == 0) {
        VQAsmHdr* h = reinterpret_cast<VQAsmHdr*>(out);
        h->n = (unsigned long long)n;
        h->err = *d.error;
        d.pref[d.nwords / 4 + kAsmCtas] = (unsigned)n;
    }
    // the columns' end: the last CTA's, when all of its warps are through
    if (d.clk && d.write) {
        __syncthreads();
        if (tid == 0 && atomicAdd(d.clk + VQ_CLK_DONE, 1ull) % kAsmCtas == kAsmCtas - 1) asm_clock(d, reinterpret_cast<VQAsmHdr*>(out));
    }
}

// The columns of a large table, written by the whole GPU after k_assemble has
// placed its rows.
__global__ void __launch_bounds__(256) k_asm_write(const VQAsmDesc* g, char* base) {
    __shared__ VQAsmDesc d;
    __shared__ VQAsmCol cols[kAsmMaxCols];
    for (int i = threadIdx.x; i < (int)(sizeof d / 4); i += blockDim.x) ((int*)&d)[i] = ((const int*)g)[i];
    __syncthreads();
    for (int i = threadIdx.x; i < d.ncols * (int)(sizeof(VQAsmCol) / 4); i += blockDim.x) ((int*)cols)[i] = ((const int*)d.cols)[i];
    __syncthreads();
    const long long n = d.pref[d.nwords / 4 + kAsmCtas];
    asm_write(d, cols, base + d.out, min(n, d.cap_rows), (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5);
    if (!d.clk) return;
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(d.clk + VQ_CLK_DONE, 1ull) % gridDim.x == gridDim.x - 1) asm_clock(d, reinterpret_cast<VQAsmHdr*>(base + d.out));
}

int out_width(int type) { return (type == VEXQ_TYPE_INT64 || type == VEXQ_TYPE_FLOAT64) ? 8 : type == VEXQ_TYPE_BOOL ? 1 : 4; }

// Bits the NULL-keyed groups' rows take ahead of the others (0: one phase).
long long phase_span(const Plan& p, long long row0, long long row1) {
    bool null_keys = false;
    for (const KeyCol& k : p.keys) null_keys = null_keys || k.nullable;
    return p.intkey_order && null_keys ? row1 - row0 : 0;
}
long long bitmap_words(const Plan& p, long long row0, long long row1) {
    const long long bits = (row1 - row0) + phase_span(p, row0, row1);
    return (bits / 32 + 4) & ~3LL;
}

}  // namespace

bool asm_plan_ok(const Plan& p) {
    // joins order groups by (probe row, chain position), which no row bitmap
    // holds; string MIN/MAX map ranks back to strings on the host; HAVING and
    // ORDER BY take the groups unordered
    if (p.path == AggPath::Regs || p.is_join || p.keys.empty()) return false;
    if (p.having_root >= 0 || p.order.sort_col >= 0) return false;
    if (p.keys.size() + p.outs.size() > (size_t)kAsmMaxCols) return false;
    for (const AggOut& a : p.outs)
        if (a.rank_dict) return false;
    return true;
}

// Tables of up to 2^20 slots and scans of up to 2^28 rows: one cluster passes
// over the slots twice and over a bit a row three times. 1,000,000 groups take 634
// us behind the scan, most of it their way over PCIe (a run 0.70 ms; 120 ms with
// the compaction over the whole GPU and the host's ordering). 4,000 groups of 2^24,
// 2^26 and 2^28 rows take 29, 74 and 242 us (runs 74, 191 and 631; by the other
// way 424, 473 and 754): about where one cluster's passes over the bits cost what
// they save.
bool asm_run_ok(const Plan& p, long long nslots, long long row0, long long row1) {
    return asm_plan_ok(p) && nslots <= (1LL << 20) + 1 && row1 - row0 <= (1LL << 28);
}

AsmLayout asm_layout(const Plan& p, long long cap) {
    AsmLayout L;
    size_t off = sizeof(VQAsmHdr);
    auto take = [&](size_t b) {
        const size_t o = off;
        off += (b + 127) & ~(size_t)127;
        return (long long)o;
    };
    auto place = [&](VQAsmCol& c, int type) {
        c.width = out_width(type);
        c.vals = take((size_t)cap * c.width);
        c.valid = take((size_t)(cap + 31) / 32 * 4);
        L.cols.push_back(c);
    };
    unsigned long long stride = 1;
    for (const KeyCol& k : p.keys) {
        VQAsmCol c;
        std::memset(&c, 0, sizeof c);
        c.nullable = k.nullable;
        c.domain = k.domain > 0 ? (unsigned long long)k.domain : 0ull;
        c.vmin = k.type == VEXQ_TYPE_DATE || k.type == VEXQ_TYPE_INT64 ? k.vmin : 0;
        if (k.domain <= 0) c.vmin = 0;
        c.nn = -1;
        if (p.path == AggPath::Hash) {
            c.src = ASM_PACKED_KEY;
            c.shift = k.shift;
            c.bits = k.bits;
            c.date33 = k.domain <= 0 && k.type == VEXQ_TYPE_DATE;
        } else {
            c.src = ASM_DENSE_KEY;
            c.stride = stride;
            stride *= c.domain ? c.domain : 1;
        }
        place(c, k.type);
    }
    for (const AggOut& a : p.outs) {
        VQAsmCol c;
        std::memset(&c, 0, sizeof c);
        const Slot& sl = p.slots[a.value_slot];
        c.slot = p.slot_pos[a.value_slot];
        c.nn = a.kind == VEXQ_AGG_COUNT ? -1 : p.slot_pos[a.nn_slot];
        c.src = a.kind == VEXQ_AGG_COUNT ? ASM_INT
              : a.kind == VEXQ_AGG_AVG ? ASM_AVG
              : sl.kind == S_FSUM ? ASM_FSUM
              : sl.kind == S_FMIN || sl.kind == S_FMAX ? ASM_FKEY : ASM_INT;
        place(c, a.out_type);
    }
    L.bytes = off;
    return L;
}

size_t asm_span(const Plan& p, long long row0, long long row1, VQAsmDesc& d) {
    d.row0 = row0;
    d.phase_bits = phase_span(p, row0, row1);
    d.nwords = bitmap_words(p, row0, row1);
    return (size_t)d.nwords * 4;
}

size_t asm_scratch(VQAsmDesc& d, long long cap, char* base) {
    d.cap_rows = cap;
    d.pref = (unsigned*)base;
    d.perm = d.pref + d.nwords / 4 + kAsmCtas + 1;
    return (size_t)(d.nwords / 4 + kAsmCtas + 1 + cap) * 4;
}

void asm_launch(const VQAsmDesc* d, int n, char* base, char* const* basep, cudaStream_t s) {
    k_assemble<<<n * kAsmCtas, kAsmThreads, 0, s>>>(d, base, basep);
    VQ_CUDA(cudaGetLastError());
}

void asm_launch_write(const VQAsmDesc* d, char* base, cudaStream_t s) {
    k_asm_write<<<2 * sm_count(), 256, 0, s>>>(d, base);
    VQ_CUDA(cudaGetLastError());
}

vexq_result_s* asm_result(Plan& p, const AsmLayout& L, const char* data, long long n, const std::shared_ptr<OutBlock>& blk) {
    auto r = std::make_unique<vexq_result_s>();
    if (p.order.limit >= 0 && p.order.limit < n) n = p.order.limit;
    r->nrows = n;
    r->block = blk;
    if (!blk) {
        auto own = std::make_shared<OutBlock>();
        size_t bytes = 0;
        for (const VQAsmCol& c : L.cols) bytes += (((size_t)n * c.width + 7) & ~(size_t)7) + (((size_t)n + 7) / 8 + 7 & ~(size_t)7);
        own->heap.reset(new char[std::max<size_t>(bytes, 1)]);
        r->block = own;
    }
    size_t at = 0;
    auto keep = [&](long long off, size_t bytes) -> const char* {
        if (blk) return data + off;
        char* to = r->block->heap.get() + at;
        std::memcpy(to, data + off, bytes);
        at += (bytes + 7) & ~(size_t)7;
        return to;
    };
    for (size_t i = 0; i < L.cols.size(); i++) {
        OutColumn oc;
        const bool key = i < p.keys.size();
        const VQAsmCol& c = L.cols[i];
        if (key) {
            const KeyCol& k = p.keys[i];
            const Column& col = p.t->cols[k.col];
            oc.name = k.name.empty() ? col.name : k.name;
            oc.type = k.type;
            if (k.type == VEXQ_TYPE_STRING) oc.flat = flat_dict(col);
            oc.distinct = p.keys.size() == 1;  // the only key: every group has a value of its own
        } else {
            const AggOut& a = p.outs[i - p.keys.size()];
            oc.name = a.name;
            oc.type = a.out_type;
        }
        oc.dv = keep(c.vals, (size_t)n * c.width);
        oc.dm = (const uint8_t*)keep(c.valid, ((size_t)n + 7) / 8);
        r->cols.push_back(std::move(oc));
    }
    return r.release();
}

}  // namespace vq
