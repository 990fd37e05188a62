// The plain FP64 form's sums over samples as integer products on the tcgen05
// tensor cores (contract_i8.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace scp3 {
namespace i8 {

// Kinds of table entries: kind | a << 4 | b << 6 | mode << 8
enum : uint32_t { kOne = 0, kHo = 1, kKa0 = 2, kV = 3, kKab = 4 };
constexpr uint32_t kZeroRow = 0xffffffffu;   // padding row: digits zero since creation, never written
constexpr int kMaxTable = 1024;              // table entries (10-bit indices)
constexpr int kKB = 64;                      // samples per k-block

// One operand array of `rows` rows (a multiple of 128): row r is the product of
// three table entries (xdesc, 10-bit indices; entry 0 is the constant 1).  With
// dual = D > 0, row D + r is V times row r for r < D (rows = 2 D).  xdesc holds the
// rows before `dual` (or all of them), then nsum rows that are only summed.
struct Plan {
    int rows = 0, dual = 0, nsum = 0, nm = 0, trows = 0;
    int ntiles = 0, nsplit = 1, sms = 148;
    int half_tiles = 0;            // tiles of one B panel
    int64_t chunk = 0, nkb = 0;    // samples and k-blocks of a whole pass
    uint8_t* x = nullptr;          // [row block][k-block][digit 1..7][128 x 64]
    int* rowmax = nullptr;         // [rows] high word of the row's largest |value| of the pass, then limits, heavy
    int v_entry = -1;              // table entry of V, -1 = none
    int scan_per = 0;              // rows per CTA of the scan
    int16_t* entries = nullptr;    // [nm][12] table entry of each kind of each mode, -1 = none
    uint32_t *xdesc = nullptr, *tspec = nullptr;     // row descriptors, then table entries
    // samples left out of the digits and added in FP64 (contract_i8.cu, "Range"): the
    // pass's limits of V, q and dV/dq (high words), a bit per sample, whether there are any
    int* limits = nullptr;         // [1 + 2 nm]
    uint32_t* heavy = nullptr;     // [chunk / 32], then any
    int4* tiles = nullptr;         // (A row, B rows 0..127, 1 = that panel only, B rows 128..255)
    double* partial = nullptr;     // [nsplit][ntiles][128 x 256] tile-local column-major
    double* spart = nullptr;       // [blocks of the scan][nsum]
    double* sums = nullptr;        // [nsum]
    // per unit (split, tile): whether its partial holds sums.  Resetting clears these
    // instead of the partials, whose first drain stores; read-outs skip the other units
    // (dimer, 2^14 samples: 151 us a pass, now 141; hexamer gradient 7893, now 7833).
    int* filled = nullptr;         // [nsplit][ntiles], then err
    int* err = nullptr;            // a bounded wait expired
};

// Table entries and rows of the direct estimator's operand: the basis functions of
// `desc`, for a plan with dual = nb_pad.
void direct_rows(const std::vector<uint32_t>& desc, int nm, int nb_pad, std::vector<uint32_t>& tspec,
                 std::vector<uint32_t>& xdesc);
int create(Plan& p, const std::vector<uint32_t>& tspec, const std::vector<uint32_t>& xdesc, int rows, int dual,
           int nsum, int nm, const std::vector<int4>& tiles, int nsplit, int64_t chunk, int sms);
void destroy(Plan& p);
int zero(const Plan& p, cudaStream_t s);
// Samples of a pass holding nvalid samples (padding samples carry V = 0 and dV/dq = 0).
inline int64_t pass_samples(int64_t nvalid) { return (nvalid + kKB - 1) / kKB * kKB; }
// The digits of a pass of k samples (vq may be null), then its products into the partials
// (of the same arrays).  Passes of few samples are added in FP64 by contract() alone.
int prepare(const Plan& p, const double* q, const double* v, const double* vq, int64_t k, cudaStream_t s);
int contract(const Plan& p, const double* q, const double* v, const double* vq, int64_t k, cudaStream_t s);
int plan_splits(int ntiles, int64_t chunk, int sms);   // sample ranges per tile of a pass
int few_ranges(int ntiles, int half_tiles, int nsplit, int nsum, int sms, int64_t k);
int table_room();                                     // table entries that fit a CTA
int check(const Plan& p, cudaStream_t s);   // synchronises; SCP3GPU_ERR_TIMEOUT after an expired wait

}  // namespace i8
}  // namespace scp3
