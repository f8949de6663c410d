// qs_sweep.h — programs of the gradient sweeps: a tiled stage's gates as passes over a tile.
//
// The forward run of a parameterised circuit and the adjoint's reverse walk take a stage's gates in
// three kinds of passes over the tile in shared memory (qs_sweep.cuh):
//   rotations  an RX or RY gate on each of the 1..3 tile bits a thread holds in registers
//   moves      a run of CNOT, X and SWAP gates, which together read amplitude x from one affine index
//              f(x) = M x ^ v over GF(2), with the run of RZ gates before or behind it, which together
//              multiply by one phase per amplitude
//   fixed      any other gate, on its own
// Gates change places only where they share no qubit.
#pragma once

#include <stdint.h>

#include <vector>

#include "qs_tile.h"

namespace qs {

constexpr int kSwMaxT = 11;        // tile qubits
constexpr int kSwMaxPass = 64;     // passes of a program
constexpr int kSwMaxDiag = 6;      // of them with phases (their factor tables stay in shared memory)
constexpr int kSwMaxRot = 64;      // rotations of a program (their sums stay in shared memory)
constexpr int kSwOutside = 6;      // controls outside the tile of one pass's moves

enum SwKind : uint8_t { SW_ROT = 0, SW_MOVE = 1, SW_FIXED = 2 };

// Register bits of a tuple: 2^rb amplitudes of a vector per thread. Smaller tiles take fewer, so that at
// least four warps (one per SM sub-partition) share a tile of 8 qubits. (Four amplitudes per thread and 512
// threads on complex128 tiles of 11 qubits: 5.19 ms for a 20-qubit gradient against 4.63 ms.)
constexpr int sw_register_bits(int T) { return T >= 10 ? 3 : T == 9 ? 2 : 1; }

struct alignas(16) SweepPass {
    uint8_t kind;
    uint8_t nout;         // SW_MOVE: entries of oq / om
    int8_t diag;          // SW_MOVE: index of its factor table, -1: no phases
    uint8_t phase_first;  // SW_MOVE, forward: the phases come before the move (read at f(x)), else behind it
    uint8_t moves;        // SW_MOVE: f is not the identity
    uint8_t rx;                  // SW_ROT: the register bits whose rotation is an RX
    int8_t rot[3];               // SW_ROT: program-local rotation on register bit j, -1: none
    uint8_t rbit[3];             // SW_ROT: tile bit of register bit j (ascending)
    int8_t zrot[kSwMaxT];        // SW_MOVE: program-local rotation of the RZ on tile bit b, -1: none
    uint8_t oq[kSwOutside];      // SW_MOVE: the bits of v set by qubit oq[i] outside the tile ...
    uint16_t om[kSwOutside];     // ... are om[i]
    uint16_t col[kSwMaxT];       // SW_MOVE: column b of M
    uint16_t flip;               // SW_MOVE: the constant part of v
    int32_t op;                  // SW_FIXED: index of its TileOp
    uint32_t seg[4];             // SW_ROT: tuple p sits at OR_j (p << j) & seg[j]
};

// One stage's program: its passes and, per program-local rotation, the index of its coefficients.
struct SweepProgram {
    std::vector<SweepPass> passes;
    std::vector<int> rots;       // program-local rotation -> the caller's gate index
    int ndiag = 0;
};

// A gate of a stage as the builder takes it, in execution order.
struct SweepGate {
    int gate = 0;                // the caller's index
    int axis = 0;                // QS_GATE_RX / RY / RZ, 0: fixed
    int target = 0;              // rotation's qubit
    const OpDesc* fixed = nullptr;
};

// The programs of one stage (several when a limit above is met), its fixed gates appended to *ops, for
// fixed-point or floating tiles, in the forward run or the reverse walk. ordered: gates keep their order
// (with a gate that is not unitary among them, an inner product depends on what was un-applied before).
std::vector<SweepProgram> build_sweep(const std::vector<SweepGate>& gates, const TileStage& st, bool fixed_point,
                                      bool reverse, bool ordered, std::vector<TileOp>* ops);

// Whether a 2^k x 2^k matrix is unitary (to 1e-9): the gates of fixed-point tiles have to keep norms.
bool is_unitary(const double* m, size_t k);

// Whether complex128 tiles are fixed point. Their error is 2^-60 of the tile's norm on every component, so amplitudes
// far below the norm, and derivatives that hang on them, lose relative accuracy: QS_ARITH_EXACT, what a register starts
// with, holds them in FP64 (8, 16, 20 qubits: 270, 940, 7070 us against 196, 768, 3890 us in fixed point).
inline bool sweep_fixed_point(int arith, bool unitary) { return unitary && arith != QS_ARITH_EXACT; }

// A rotation's coefficients on the device, for every tile type (sweep_coefs in qs_sweep.cuh fills them
// from the angle).
//   floating tiles, RX and RY: the pair update without its common factor f (a' = a + t b and so on: two
//     multiply-adds per real pair instead of four operations) in the form with |t| <= 1: c = t = tan
//     (f = cos), s = 0; or behind an exchange of the pair c = t = -cot (f = sin), s = 1
//   RZ: c = cos, s = sin of theta / 2, and the same as 2^60 ths in limbs (complex64: as float pairs)
//   fixed-point tiles, RX and RY: theta / 2 = a + k pi / 2 with |a| <= pi / 4, the rotation by a as three
//     shears with tan(a / 2) and sin(a), as 2^60 ths in limbs; `quarter` for odd k
struct alignas(16) SweepCoef {
    double c, s;
    int32_t ph, pl, sh, sl;  // limbs of -tan(a / 2) and sin(a); RZ: of cos and sin
    long long pk, sk;        // what rounds the limb products (FxLimb)
    int32_t quarter, pad[3];
};

}  // namespace qs
