// What a batch takes of the device's memory: the engine's attach sizes its buffers by it, and the
// job server admits jobs by it.  Host code without CUDA.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>

namespace pdpd {

// Room for the FP64 engine's pair lists: candidates and the pairs that its beads evaluate
// themselves (half of those, and both sides of the pairs across the box's faces), at each world's
// mean density with a margin for its fluctuations.  Beads that find no room are evaluated without
// lists, with the same result.
struct List64Room {
    double entries = 0, pairs = 0;
    // one buffer: cursors, a record per bead, entries, pairs, terms
    size_t off_lrec() const { return 256; }
    size_t off_list(size_t n_beads) const { return off_lrec() + up(8 * n_beads); }
    size_t off_pairs(size_t n_beads) const { return off_list(n_beads) + up(4 * (size_t)entries); }
    size_t off_term(size_t n_beads) const { return off_pairs(n_beads) + up(8 * (size_t)pairs); }
    size_t bytes(size_t n_beads) const { return off_term(n_beads) + up(24 * (size_t)pairs); }
    static size_t up(size_t n) { return (n + 255) & ~size_t(255); }
    void add(double n, const int32_t box[3], bool asym)
    {
        const double near = 1.3 * 4.19 * n / ((double)box[0] * box[1] * box[2]);
        double across = 0;
        for (int k = 0; k < 3; k++) across += 0.375 / box[k];
        entries += n * (near + 8);
        pairs += n * (near * (asym ? 1.0 : 0.5 + 0.5 * std::min(1.0, across)) + 5);
    }
};

// What the lists save over the force pass without them (k_force64), us a step, for a world of n
// beads: the list kernel goes through all cells, at 0.088 ns each; without lists
// the FP64 work grows with the density, and beyond about 4 beads a cell its candidate lists
// overflow.  Steps of water boxes, us, with lists and without: 64^3 of density 0.05 54 and 41, 0.1 59
// and 49, 0.2 65 and 73, 3 833 and 1,771; 90^3, 0.2 149 and 116, 0.25 159 and 133, 0.3 172 and 176;
// 128^3, 0.05 267 and 89, 0.2 370 and 275, 0.25 405 and 345, 0.3 447 and 466; 160^3, 0.25 775 and 679,
// 0.3 837 and 878; 24^3, 10 657 and 14,400.  A world costs the list kernel a brick at least, about
// 120 cells' worth: 2,000 boxes of 2^3 of density 0.25 74 and 59, 0.5 82 and 80, 1 94 and 116.  And
// bricks that a world does not fill cost more for each of its cells, which the mean of its cells
// and the cells of its 5x8x8 bricks describes: 100 boxes of 11x9x14 (3,840 for 1,386) of density
// 0.05 57 and 39, 0.15 62 and 46; 1,000 of 6^3 (640 for 216), 0.15 94 and 68, 0.4 118 and 110; 1,000
// of 8^3 (640 for 512), 0.25 131 and 111; ten of 24^3 (14,400 for 13,824), 0.05 45 and 41, 0.25 50 and
// 60.
inline double lists64_saving_us(double n, const int32_t box[3])
{
    const double cells = (double)box[0] * box[1] * box[2];
    const double padded = 320.0 * ((box[0] + 4) / 5) * ((box[1] + 7) / 8) * ((box[2] + 7) / 8);
    const double rho = n / cells;
    const double bead_ns = rho > 3 ? 1.2 * std::pow(rho / 3, 3) : std::min(1.2, 1.1 * rho);
    return 1e-3 * (n * bead_ns - 0.088 * std::max(std::sqrt(cells * padded), 120.0));
}
// Small batches gain at any density: a bead's walk on global memory is a long chain (32^3 of
// density 0.005 to 0.1 30 to 33 with lists, 34 to 40 without; 50^3, 0.05 43 and 39).
constexpr double LISTS64_BASE_US = 12;
// And the chain is the longer the denser the densest world, however few its beads: 63x53x91 of density
// 0.11 and 10x9x8 of density 3, 73 with lists and 99 without, and 6^3 of density 1 67 and 62; 90^3 of
// density 0.2 and 6^3 of density 3, 153 and 166, and 1 150 and 126.
inline double lists64_chain_us(double most_density)
{
    return 25 * std::min(1.0, std::max(0.0, (most_density - 0.4) / 1.6));
}

// Entries of a cell's bucket in a world of this density: the mean and 5.5 Poisson deviations (cells
// that hold more go through overflow lists), a multiple of 4.
inline uint32_t bucket_room(double density)
{
    return (uint32_t)(4 * std::ceil((density + 5.5 * std::sqrt(density) + 3) / 4));
}

// Device bytes per bead: state A and B (3 + 3 vectors), ids, cells, slots by id, keys, two rows of 9
// doubles in id order, hashes twice, polymer-bead list, scratch, overflow node, bond row; FP32 bond
// forces or FP64 cell offsets.
constexpr size_t BEAD_BYTES32 = 6 * 16 + 16 + 144 + 8 + 4 + 4 + 8 + 4 + 16;
constexpr size_t BEAD_BYTES64 = 6 * 32 + 16 + 144 + 8 + 4 + 4 + 8 + 4 + 16;

// The sizes of a batch's worlds, added up.
struct BatchSize {
    uint64_t worlds = 0, beads = 0, cells = 0, bucket_entries = 0, bonds = 0, angles = 0;
    List64Room room;
    double saving_us = LISTS64_BASE_US;  // of the pair lists, but for the chain
    double most_density = 0;

    void add(uint32_t n_beads, const int32_t box[3], uint32_t n_bonds, uint32_t n_angles, bool asym)
    {
        const uint64_t c = (uint64_t)box[0] * box[1] * box[2];
        worlds++;
        beads += n_beads;
        cells += c;
        bucket_entries += c * bucket_room((double)n_beads / (double)c);
        bonds += n_bonds;
        angles += n_angles;
        if (n_beads) room.add((double)n_beads, box, asym);
        saving_us += lists64_saving_us((double)n_beads, box);
        most_density = std::max(most_density, (double)n_beads / (double)c);
    }
    void add(const BatchSize &o)
    {
        worlds += o.worlds;
        beads += o.beads;
        cells += o.cells;
        bucket_entries += o.bucket_entries;
        bonds += o.bonds;
        angles += o.angles;
        room.entries += o.room.entries;
        room.pairs += o.room.pairs;
        saving_us += o.saving_us - LISTS64_BASE_US;
        most_density = std::max(most_density, o.most_density);
    }

    // Entries of every bucket of the batch: as many in all as the worlds' own sizes come to, so that a
    // few dense worlds do not make every cell of the others as large (their cells overflow more
    // often then, with the same result).
    uint32_t bucket_k() const { return cells ? std::max<uint32_t>(4, (uint32_t)(bucket_entries / cells) & ~3u) : 4u; }

    // The pair lists can address the batch (a list entry holds a slot in 25 bits, a pair in 30), and
    // save time.
    bool lists_fit() const { return beads > 0 && beads < (1u << 25) && room.entries < 2e9 && room.pairs < 1e9; }
    bool lists_pay() const { return saving_us + lists64_chain_us(most_density) > 0; }

    // Device bytes of the batch.
    size_t bytes(bool fp64) const
    {
        size_t n = (fp64 ? BEAD_BYTES64 : BEAD_BYTES32) * beads + (20 + 4 * (size_t)bucket_k()) * cells +
                   48 * (2 * bonds + 3 * angles) + 4096 * worlds;
        if (fp64 && lists_fit() && lists_pay()) n += room.bytes(beads);
        return n;
    }
};

// Whether a job joins a running batch (its size, 0 worlds: none) within the budget.  An FP64 batch
// is kept small enough for its pair lists: without them its steps take about twice as long.
inline bool job_joins(const BatchSize &batch, const BatchSize &job, bool fp64, size_t budget)
{
    if (batch.worlds == 0) return true;
    BatchSize all = batch;
    all.add(job);
    if (all.bytes(fp64) > budget) return false;
    return !(fp64 && all.lists_pay() && !all.lists_fit() && batch.lists_fit());
}

// Bytes of a host snapshot buffer (rows x, v, f as doubles) for the batches that a budget admits.
// FP64: no batch with pair lists takes less than 600 bytes a bead, nor has 2^25 beads; a single
// job that is larger gets a larger buffer when it comes.
inline size_t snapshot_reserve(bool fp64, size_t budget)
{
    const size_t beads = fp64 ? std::min<size_t>(budget / 600, size_t(1) << 25) : budget / BEAD_BYTES32;
    return std::min<size_t>(9 * sizeof(double) * beads, size_t(16) << 30);
}

}  // namespace pdpd
