// Compiles plans against tables that have a schema and no rows in memory, for
// tests on hosts without a GPU: the library generates and compiles a plan's
// kernels there and leaves them unloaded. Built and called by plan_probe.py.
#include <cstring>
#include <sstream>
#include <string>

#include "plan.h"

using namespace vq;

namespace {

int put(const std::string& s, char* out, int cap) {
    std::strncpy(out, s.c_str(), cap - 1);
    out[cap - 1] = 0;
    return s.rfind("error ", 0) == 0 ? -1 : 0;
}

std::string show(const Plan& p) {
    std::ostringstream o;
    o << "lsb=";
    for (size_t i = 0; i < p.fx_lsb.size(); i++) o << (i ? "," : "") << p.fx_lsb[i];
    int sums = 0;  // places the main kernel's text adds a warp's float sum
    for (size_t at = 0; (at = p.src_main.find("vq_w_fx_add<", at)) != std::string::npos; at++) sums++;
    o << " warp_sums=" << sums << " " << p.explain;
    return o.str();
}

}  // namespace

extern "C" {

struct ProbeColumn {
    int32_t type, nullable, has_range, finite;
    int64_t dict, imin, imax;  // dict: entries of a STRING column's dictionary
    double fmin, fmax;
};

void* probe_table(int n, const ProbeColumn* c, int64_t nrows) {
    Table* t = new Table;
    t->nrows = nrows;
    t->n_rg = (int32_t)((nrows + t->rg_rows - 1) / t->rg_rows);
    t->cols.resize(n);
    for (int i = 0; i < n; i++) {
        Column& k = t->cols[i];
        k.name = "c" + std::to_string(i);
        k.type = c[i].type;
        k.nullable = c[i].nullable;
        k.has_range = c[i].has_range;
        k.finite = c[i].finite;
        k.imin = c[i].imin;
        k.imax = c[i].imax;
        k.fmin = c[i].fmin;
        k.fmax = c[i].fmax;
        for (int64_t d = 0; d < c[i].dict; d++) k.dict.add("s" + std::to_string(d));
    }
    return t;
}

void probe_table_free(void* t) { delete (Table*)t; }

int probe_agg(void* t, const vexq_agg_plan_desc* d, char* out, int cap) {
    try {
        std::unique_ptr<Plan> p(compile_agg((Table*)t, d));
        return put(show(*p), out, cap);
    } catch (const std::exception& e) {
        return put(std::string("error ") + e.what(), out, cap);
    }
}

// The key a Filter call's plan is kept under: its length, and the key's bytes in out.
int probe_filter_key(void* t, const vexq_expr* nodes, int nnodes, const int32_t* children, int nchildren, int pred, char* out, int cap) {
    try {
        SelectLease l(*(Table*)t, 'f', nodes, nnodes, children, nchildren, pred, nullptr, 0);
        std::memcpy(out, l.key.data(), std::min<size_t>(l.key.size(), cap));
        return (int)l.key.size();
    } catch (const std::exception& e) {
        return put(std::string("error ") + e.what(), out, cap);
    }
}

// Pinned bytes a pool holds after n blocks of `bytes` were taken and kept, and
// (in lent) how many of them results may keep. Needs a GPU.
int64_t probe_out_pool(int n, int64_t bytes, int64_t lend_most, int32_t* lent) {
    try {
        OutPool pool;
        pool.lend_most = (size_t)lend_most;
        std::vector<std::shared_ptr<OutBlock>> held;
        *lent = 0;
        for (int i = 0; i < n; i++) {
            bool lend = false;
            std::shared_ptr<OutBlock> b = pool.acquire((size_t)bytes, lend);
            if (b && lend) {
                held.push_back(b);
                ++*lent;
            }
        }
        return (int64_t)pool.bytes();
    } catch (const std::exception&) {
        return -1;
    }
}

// The kernel for group tables too large for a slot and a sign in a word, for a
// plan compiled here or (probe_widen) a prepared one.
int probe_agg_wide(void* t, const vexq_agg_plan_desc* d, char* out, int cap) {
    try {
        std::unique_ptr<Plan> p(compile_agg((Table*)t, d));
        widen_slots(*p);
        return put(show(*p), out, cap);
    } catch (const std::exception& e) {
        return put(std::string("error ") + e.what(), out, cap);
    }
}

int probe_widen(vexq_plan_s* h) {
    try {
        widen_slots(*h->p);
        return 0;
    } catch (const std::exception&) {
        return -1;
    }
}

int probe_join(void* build, void* probe, const vexq_join_plan_desc* d, char* out, int cap) {
    try {
        std::unique_ptr<Plan> p(compile_join((Table*)build, (Table*)probe, d));
        return put(show(*p), out, cap);
    } catch (const std::exception& e) {
        return put(std::string("error ") + e.what(), out, cap);
    }
}
}
