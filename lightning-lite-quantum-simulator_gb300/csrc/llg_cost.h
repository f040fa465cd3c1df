// llg_cost.h -- what gate lists cost in the two forms of a plan, tile passes and dense 5-qubit blocks: the rates that the
// choices of a state's flush (llg_engine.cu), of a batch (llg_batch.cu) and of the adjoint sweeps (llg_adjoint.cu) are made
// with.  All measured on this GPU.
#pragma once

#include <algorithm>
#include <cmath>

#include "../../include/llgpu.h"
#include "llg_internal.h"

namespace llg {

// FP64 tile passes of large registers: multiply-adds a second, and an amplitude for a merged one-qubit gate that mixes
constexpr double kTileFmaRate = 0.56e12, kTileMixFma = 3.2;
// seconds an amplitude: a pass that only moves or signs (2.6 ms per 2^30)
constexpr double kSingleAmp = 2.4e-12;

// Microseconds that tile passes take for a gate on 6 .. 12 qubits, where a CTA's latency and not the arithmetic counts: fits of
// 20 lists a size (random H, RY, 2x2s or rotations with 1/4 and 1/2 CNOTs, layers of rotations and CNOTs or CZs, CNOTs alone),
// most within 20 %; dense random 2x2s take up to twice what is written here.  Sign flips join the phases beside them.
struct TileGates {
    double h, real, general, diag, move;
};
inline TileGates tile_latency(int P, int n) {
    static constexpr TileGates f64[7] = {{1.2, 1.0, 1.3, 1.1, 0.57},  {1.15, 1.05, 1.4, 1.35, 0.56}, {1.15, 1.15, 1.55, 1.5, 0.55},
                                         {1.5, 1.5, 2.1, 2.6, 0.57},  {2.4, 2.35, 3.1, 4.5, 0.73},   {4.1, 3.85, 4.7, 7.0, 1.05},
                                         {7.3, 7.2, 8.0, 10.0, 1.64}};
    static constexpr TileGates df64[7] = {{0.82, 0.75, 1.1, 0.95, 0.42}, {0.78, 0.78, 1.2, 1.2, 0.40}, {0.8, 0.87, 1.4, 1.5, 0.40},
                                          {0.9, 1.05, 1.8, 2.6, 0.42},   {1.2, 1.5, 2.55, 4.5, 0.51},  {1.85, 2.4, 4.0, 7.0, 0.63},
                                          {2.4, 4.5, 6.4, 10.0, 0.78}};
    const int i = std::min(std::max(n, 6), 12) - 6;
    return P == LLG_F64 ? f64[i] : df64[i];
}

// Tile passes for these gates: their latencies (15 % more on several CTAs) and arithmetic (a CNOT between random qubits takes
// 38 us at 2^24 amplitudes in FP64, 18.6 in double-float), at least one read and write of the state; channels are sparse
// passes of their own, 6.2 ms per 2^30 on one qubit of a density matrix, 9 on two, at least 6 us.
inline double tile_latency_seconds(int P, int n, const GateCounts& c) {
    const TileGates l = tile_latency(P, n);
    return 1e-6 * (n > 12 ? 1.15 : 1.0) *
           (l.h * c.h + l.real * c.real + l.general * c.general + l.diag * c.diag + l.move * c.moves);
}
inline double tile_arith_seconds(int P, int n, const GateCounts& c) {
    const int mixing = c.h + c.real + c.general;
    return (double)(1ULL << n) * (P == LLG_F64 ? kTileMixFma / kTileFmaRate * mixing + 2.0e-12 * c.diag + 2.3e-12 * c.moves
                                              : 2.0e-12 * mixing + 1.9e-12 * c.diag + 1.1e-12 * c.moves);
}
inline double tile_seconds(int P, int n, const GateCounts& c) {
    const double amps = (double)(1ULL << n), latency = tile_latency_seconds(P, n, c), arith = tile_arith_seconds(P, n, c);
    const double channels = c.small * std::max(6e-6, amps * 5.8e-12) + c.large * std::max(6e-6, amps * 8.4e-12);
    const bool gates = c.h + c.real + c.general + c.diag + c.moves + c.flips > 0;
    const double both = arith + latency - (P == LLG_F64 ? 0.0 : 0.5 * std::min(arith, latency));  // the FP32 pipe hides more
    return (gates ? std::max(both, amps * 4.8e-12) : 0.0) + channels;
}

// Blocks, and gates on their own between them: a block takes 8.2 us (7.6 on the 6 to 11 qubits of a part of a tile), and from 20
// qubits on 5.5 us (6.6 in double-float) for every round of the SMs over its tiles of 4096 amplitudes.
inline double block_seconds(int P, int n, double blocks, double singles) {
    const double amps = (double)(1ULL << n);
    const double rounds = std::ceil(amps / (4096.0 * 152.0));
    const double block = n < 12 ? 7.6e-6 : n < 20 ? 8.2e-6 : 4e-6 + rounds * (P == LLG_F64 ? 5.5e-6 : 6.6e-6);
    return blocks * block + singles * (3e-6 + amps * kSingleAmp);
}

// The number of blocks that a list is likely to take: 9 two-qubit gates a block where each qubit has them with a few others only
// (a chain, a ring), between random qubits 9 on 6 qubits and 5 on 10 and more, and 12 to 17 merged one-qubit gates, of five
// qubits.
inline double likely_blocks(int n, const GateCounts& c, int two, double partners) {
    static constexpr double random[] = {9.0, 7.0, 6.3, 5.6, 5.0}, merged[] = {17.0, 17.0, 13.0, 14.0, 12.0};
    const int i = std::min(std::max(n, 6), 10) - 6;
    const int one = c.h + c.real + c.general + c.diag;
    return std::max(std::ceil(std::min(n, one) / 5.0), std::max(two / (partners > 3.5 ? random[i] : 9.0), one / merged[i]));
}

// what a flush costs besides, on the host: lists that go in few passes end before their planning
constexpr double kTileBase = 25e-6, kBlockBase = 40e-6, kBlockGate = 0.06e-6;

}  // namespace llg
