// Residue form of the split-precision GEMMs (the Ozaki scheme II: Ozaki, Uchino, Imamura,
// "Ozaki Scheme II: A GEMM-oriented emulation of floating-point matrix multiplication using
// an integer modular technique", 2025): internal interface.
//
// Every FP64 operand row x is rounded to integers X = round(x 2^(bits - e)), max |x| < 2^e,
// and an integer dot product C = X Y is found from its residues modulo n pairwise coprime
// moduli m_i below 416: one BF16 GEMM per modulus over the balanced residues of X and Y
// (|r| <= 207, exact in BF16), then C by the Chinese remainder theorem.  n moduli cost n
// products where balanced digits cost s (s + 1) / 2, and no term is dropped: the result is
// the exact product of the rounded operands.  |C| <= K 2^(2 bits) < M / 2 (M the product of
// the moduli) holds for any operands, and FP32 accumulation over kChunkK inner elements
// stays below 2^24 for any residues, so there is nothing to certify but the rounding of the
// operands.
#pragma once

#include "split.h"

namespace gain {
namespace split {

constexpr int kMaxMod = 16;
constexpr int kChunkBlocks = 6;                    // k-blocks of exact FP32 accumulation:
constexpr int kChunkK = kChunkBlocks * BK;         // 384 x 207^2 + 207 < 2^24
constexpr int kResMaxBits = 56;

// pairwise coprime, largest first
constexpr int kModuli[kMaxMod] = {415, 413, 412, 411, 409, 407, 403, 401, 397, 391, 389, 383, 379, 373, 367, 361};

// log2 of the product of the first n moduli (rounded down a little)
double residue_log2m(int n);
// The fewest moduli whose product exceeds 2 K 2^(2 bits) (0: more than kMaxMod).
int residue_moduli(int bits, int K);

// One output tile of the residue GEMM; a grouped launch lists every (tile, modulus) item.
struct ResTile {
    int m0, n0;     // first output row (relative to the launch's first) / column
    int a_k0;       // A inner coordinate of k-block 0
    int nkb;        // k-blocks of BK
    int ncols;      // 128, or (CTA pairs) 256
    int group;      // grouped launch: the item's group; -1: an empty slot of the schedule
    int mod;        // grouped launch: the item's modulus
    int pad;
};

struct ResGroup;

struct ResGemmArgs {
    const ResTile* tiles;
    int ntiles;            // single launch: every tile runs for nmod moduli, modulus by modulus
    int nmod;
    const ResGroup* groups;   // grouped launch (device memory): operands and output of each group
    int m_base;            // A row of the launch's first output row
    uint16_t* res;         // residues in [0, m_i): res[i * plane + row * ldr + col]
    long plane, ldr;
    int* err;              // device error word (0 ok, else timeout code)
    // optional: the launch's span on the global timer (ns), as maxima over the CTAs from zero:
    // span[0] the complement of the first start, span[1] the last end.  (An event between two
    // kernels costs a short run about 2 us, and the next kernel cannot be launched behind it.)
    unsigned long long* span;
};

struct alignas(128) ResGroup {
    CUtensorMap tmA, tmB;  // tmB with 64-row boxes
    uint16_t* res;
    long plane, ldr;
};

// The kernels' attributes on the current device (before a capture).
cudaError_t prepare_residue();
cudaError_t launch_residue_gemm(const CUtensorMap& tmA, const CUtensorMap& tmB, const ResGemmArgs& a, int num_sms,
                                cudaStream_t st, bool pair);
// a.tiles holds ntiles = units x k items, unit u taking items u, u + units, ...
cudaError_t launch_residue_gemm_grouped(const ResGemmArgs& a, int units, cudaStream_t st, bool pair);

// Reconstruction of the outputs from their residues, with certified bounds and flags.
struct CrtArgs {
    const uint16_t* res;
    long plane, ldr;
    int nmod, bits;
    int row0;              // output row of residue row 0
    int rows;              // residue rows to reconstruct
    int cols;              // columns to reconstruct (a multiple of 128)
    int nrow;              // rows per block (crt_set_rows; launch_crt sets it)
    int cols_valid;        // columns that are flagged and counted
    RowStats A, B;
    double* out;
    long ldo;
    float* bnd;            // optional: absolute error bound of every output
    long ldb;
    float c_fix;           // bound of the reconstruction, units of 2^{eA+eB}
    float c_f64;           // as GemmArgs
    float tol;
    int flag_mode;         // 1: bound > max(tol |value|, FP64 bound) is flagged; 2: bound > FP64 bound; 0: none
    float* rowerr2;        // optional, as GemmArgs
    unsigned long long* absmax;   // optional, as GemmArgs
    int2* flags;
    unsigned int* nflags;
    int max_flags;
    unsigned long long m_mant;    // M = m_mant 2^(m_exp - 63), 2^63 <= m_mant
    int m_exp;
};
// m_mant, m_exp and c_fix of a set of nmod moduli at `bits` fraction bits
void crt_constants(CrtArgs* a);
cudaError_t launch_crt(const CrtArgs& a, cudaStream_t st);
// Rows per block (nrow) of n reconstructions in one launch, and the blocks of one of them.
void crt_set_rows(CrtArgs* a, int n);
int crt_blocks(const CrtArgs& a);
// args[g] (device memory) runs on blocks offs[g] <= b < offs[g + 1]
struct CrtGroups {
    const CrtArgs* args;
    const int* offs;
    int n, blocks;
    int nmod;              // every group's moduli (0: they differ)
};
cudaError_t launch_crt_grouped(const CrtGroups& g, cudaStream_t st);

// Residue planes of rows (SliceArgs with bits > 0; split.h's launch_slice calls these).
cudaError_t launch_residue_slice(const SliceArgs& a, cudaStream_t st);
cudaError_t launch_residue_slice_grouped(const SliceGroups& g, bool short_rows, cudaStream_t st);

}  // namespace split
}  // namespace gain
