// assemble.h — result columns of a group table written on the device.
#pragma once

#include "plan.h"

namespace vq {

// How one output column is computed from a group's slot.
enum AsmSrc {
    ASM_DENSE_KEY = 0,  // (slot / stride) % domain, NULL = the last code of a nullable column
    ASM_PACKED_KEY,     // bits [shift, shift + bits) of the slot's key
    ASM_INT,            // integer bank entry (COUNT, integer SUM, integer / date / bool MIN and MAX)
    ASM_FSUM,           // exact float sum
    ASM_AVG,            // exact float sum ÷ non-null count
    ASM_FKEY            // float MIN / MAX from its order key
};

struct VQAsmCol {
    int src, width;     // width: bytes of a value (8, 4 or 1)
    int slot, nn;       // bank position; integer-bank position of the non-null count (-1: never NULL)
    int shift, bits;    // packed key
    int nullable, date33;  // date33: a packed date carries its NULL flag in bit 32
    unsigned long long stride, domain;
    long long vmin;
    long long vals, valid;  // byte offsets of the values and the validity bitmap in the output block
};

// Tables up to this many slots have their columns written by the cluster that
// orders them (one launch); larger ones by a second launch over the whole GPU.
constexpr long long kAsmClusterWrites = 4096;

// One group table and where its columns go.
struct VQAsmDesc {
    const unsigned long long* keys;
    const long long* first;
    const long long* acc_i;
    const long long* acc_fx;
    const unsigned* special;
    const int* fx_lsb;
    const int* error;
    unsigned long long* clk;  // the run's device clock (null: none)
    const VQAsmCol* cols;
    unsigned* bits;         // [nwords] a bit per row that is some group's first
    unsigned* pref;         // [nwords / 4 + 9] set bits before each four words, then the CTAs' totals and the group count
    unsigned* perm;         // [cap_rows] output row → slot
    long long nslots, nwords, row0, phase_bits, cap_rows;
    long long out;          // offset of the header and columns from the output base
    int ncols;
    int kst;                // words from a slot's key and first row to the next slot's
    int write;              // the cluster writes the columns too
};
struct VQAsmHdr {           // at the start of a table's output
    unsigned long long n;
    int err, pad;
    unsigned long long clk[VQ_CLK_END + 1];  // the run's device clock and the columns' end
    unsigned long long pad8;
};

// Byte layout of a plan's output columns for at most cap rows.
struct AsmLayout {
    std::vector<VQAsmCol> cols;
    size_t bytes = 0;
};

bool asm_plan_ok(const Plan& p);      // the plan's output can be assembled on the device
// … for this run: the table and the rows its order keys span
bool asm_run_ok(const Plan& p, long long nslots, long long row0, long long row1);
AsmLayout asm_layout(const Plan& p, long long cap);
// Bitmap of a scan of rows [row0, row1): its bytes. It is clear before every
// run; k_assemble clears it again after use.
size_t asm_span(const Plan& p, long long row0, long long row1, VQAsmDesc& d);
// The rest of the scratch (pref, perm) at base: its bytes.
size_t asm_scratch(VQAsmDesc& d, long long cap, char* base);
void asm_launch(const VQAsmDesc* d, int n, char* base, char* const* basep, cudaStream_t s);
void asm_launch_write(const VQAsmDesc* d, char* base, cudaStream_t s);  // the columns of a table launched with write = 0
// The result over n assembled rows at `data` (a table's output): it keeps blk,
// or its own copy of the rows when blk is null.
vexq_result_s* asm_result(Plan& p, const AsmLayout& L, const char* data, long long n, const std::shared_ptr<OutBlock>& blk);

}  // namespace vq
