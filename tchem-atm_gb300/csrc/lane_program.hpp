// Instruction streams of the batched time-advance kernel (kernels_lanes_impl.cuh).
//
// The kernel advances S samples per CTA with the sample as the fastest index of every shared-memory
// array, so the mechanism's sparse structure is the same instruction for all S samples and its
// indices are read once per S samples. The CTA's threads form P = threads / S slots; this file
// distributes the work of one Newton iteration over the slots, once per mechanism and P, as
// streams of 16-byte packets that a slot reads in order:
//
//  * matrix: the nonzeros of J and the diagonal of I - c J (the kernel zeroes the fill). One packet holds
//    two contributions (FP32: d index pair, two coefficients) or one (FP64).
//  * factor: P A P^T = L U in a static Markowitz order without pivot search, up to the last n_t
//    pivots. The pivot rows keep U unscaled, L is scaled by the pivot's reciprocal, and the diagonal
//    holds the reciprocals.
//  * the last n_t positions, where the fill has made the matrix nearly dense, are the tail: a dense
//    block that the kernel inverts in registers (Gauss-Jordan). Its triangular solves would be a
//    chain of 2 n_t levels; with the inverse they are one matrix-vector product.
//  * forward, backward: substitution with the sparse rows before and after that product.
//    Factor and substitutions are lists of "entry -= l * u" products; a packet holds a header and three.
//
// Factor and substitutions are list-scheduled: a level is a set of packets whose operands were
// completed in earlier levels, spread over the slots, with a CTA barrier after it. An entry with many
// products gathers those that are ready over several levels.
#pragma once

#include <cstdint>
#include <vector>

#include "device_tables.hpp"
#include "kernels_lanes.hpp"

namespace tchem_gb {

#ifdef __CUDACC__
#define TCHEM_GB_HD __host__ __device__
#else
#define TCHEM_GB_HD
#endif

struct Packet {
  uint32_t w[4];
};

// Header of factor and substitution packets: dst (15 bits), scale (9 bits from 16: the pivot entry
// that scales the result, or the one entry), flags; those marked "warp" are the same in all of the
// warp's packets of a round. Every packet reads, updates and writes its entry.
enum LanePacket : uint32_t {
  LP_PIVOTS = 1u << 15,   // warp: some packet is a pivot
  LP_SCALE_SHIFT = 16,
  LP_SCALED = 1u << 25,   // warp: some packet's scale is a pivot entry
  LP_LCOL = 1u << 26,     // an entry of L: its size is checked
  LP_PIVOT = 1u << 27,    // a pivot: its reciprocal is stored
  LP_CONT = 1u << 28,     // goes on with the entry of the slot's packet before it
  LP_TWO = 1u << 29,      // warp: more than one product
  LP_THREE = 1u << 30,    // warp: more than two
  LP_ONE = 1u << 31       // warp: any product
};
constexpr uint32_t kLaneWarpFlags = LP_PIVOTS | LP_SCALED | LP_ONE | LP_TWO | LP_THREE;
// Matrix packets: dst (15 bits), first and last contribution of the entry, unit diagonal.
enum LaneMatrix : uint32_t { LM_START = 1u << 15, LM_END = 1u << 16, LM_DIAG = 1u << 17 };

constexpr int kLaneMaxEntries = 1 << 15;  // entries, the zero entry and the vector section
constexpr int kLaneMaxSpecies = 511;
// Species and reactions per slot, at most: registers of the kernel.
TCHEM_GB_HD constexpr int lane_species(int P) { return P == 16 ? 4 : (P == 128 ? 3 : 2); }
TCHEM_GB_HD constexpr int lane_reactions(int P) { return P == 16 ? 12 : (P == 128 ? 8 : (P < 128 ? 6 : 4)); }
constexpr int kLaneSegments = 4;  // net-production segments in the table, >= lane_species

// The tail's rows and columns are dealt to a grid of rows(P) x cols(P) slots.
TCHEM_GB_HD constexpr int lane_grid_cols(int P) { return P >= 256 ? 16 : (P >= 64 ? 8 : 4); }
// A tail row's entries lie lane_tail_stride apart from the next row's: odd, so that the rows of
// neighbouring slots start in different banks (with 16 samples two slots share a warp, the conflict is
// two-way at most, and the padding could cost the second CTA per SM).
TCHEM_GB_HD constexpr int lane_tail_stride(int P, int n_t) { return P > 16 ? n_t | 1 : n_t; }
TCHEM_GB_HD constexpr int lane_grid_rows(int P) { return P / lane_grid_cols(P); }
// Tile heights (rows per slot) that the kernel has for a slot count: n_t = height x grid rows. Widths are
// even: the kernel takes pivots in pairs.
constexpr int kLaneTiles = 4;
TCHEM_GB_HD constexpr int lane_tile(int P, int warps, int k) {
  return P >= 256 ? (k == 0 ? 2 : k == 1 ? 4 : k == 2 || warps > 8 ? 8 : 10)  // 10 x 10 takes over 128 registers
                  : P >= 128 ? k + 1 : P >= 64 ? 2 * (k + 1) : P >= 32 ? k + 1 : 2 * (k < 2 ? k + 1 : 3);
}

// Packets of each warp in turn, [rounds of the warp][slots per warp], and for the scheduled streams
// each warp's rounds per level, [level][warp] (FP32 factor: even numbers, the kernel works on two at a
// time; a warp without work goes straight to the level's barrier). A spare pair of rounds follows each
// warp's packets, for the read-ahead.
struct LaneStream {
  std::vector<int32_t> first, rounds;  // [warps]: first packet, rounds
  int levels = 0;
  std::vector<uint8_t> level_rounds;
  std::vector<Packet> packets;
};

struct LaneProgram {
  int m = 0, R = 0, P = 0;
  int nps = 0, nrs = 0;          // species and reactions per slot
  int n_t = 0, tail = 0;         // tail size (0: none) and its first entry
  // entries: pivots of the positions before the tail, the one entry (their number), the others, the
  // tail block, the zero entry, the vector section (by position)
  int zero = 0, vec = 0, n_entries = 0;
  std::vector<int32_t> species;   // [nps][P] position | species << 16 of slot p, or m
  // [nrs] rounds: reactant positions a | b << 16, c | count << 16, first d slot, reaction
  LaneStream reactions;
  LaneStream net;                 // net production: one segment per species of the slot
  std::vector<int32_t> net_end;   // [warps][kLaneSegments] rounds up to the end of each segment
  LaneStream matrix, factor, forward, backward;
};

// What a problem is made of: reactions with their reactant factors, rows of the right-hand side as sums
// over q (the reactions' rates and rows that the kernel computes otherwise), entries of the Jacobian as
// sums over d (one slot per reactant factor, and further ones).
struct LaneInput {
  int m = 0, R = 0, Q = 0, D = 0;                // rows, reactions, rows of q, slots of d
  int max_factors = 0;
  std::vector<int32_t> rf_ptr, rf_sp;            // factors of reaction r; slot numbers as d
  std::vector<std::vector<std::pair<int, double>>> net;  // [m]: (row of q, coefficient)
  struct Entry {
    int row, col;
    std::vector<std::pair<int, double>> terms;   // (slot of d, coefficient)
  };
  std::vector<Entry> jac;
  std::vector<double> emis;                      // [m]
};
LaneInput lane_input(const HostTables& ht);

// Fill and static order of a problem's Newton matrix.
struct LanePattern {
  int m = 0;
  std::vector<int32_t> order, pos;
  std::vector<char> fill;  // [m * m] by position
};

// Throws std::domain_error where the encoding does not cover the mechanism.
LanePattern build_lane_pattern(const LaneInput& in);
// The tail size for a shape, and the program.
int lane_tail_size(const LaneInput& in, const LanePattern& pat, const LaneShape& shape, bool fp64);
LaneProgram build_lane_program(const LaneInput& in, const LanePattern& pat, int P, int warps, int n_t, bool fp64);
// Entries (pattern, tail block, zero, vector section) for a tail size, without building the program.
int lane_entries(const LanePattern& pat, int P, int n_t);

}  // namespace tchem_gb
