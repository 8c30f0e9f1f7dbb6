// Host side of the LU panels on thread-block clusters: how many CTAs a panel takes.
#pragma once

#include <algorithm>
#include <cstddef>

namespace tcu {

constexpr int PC_T = 256;     // threads, and most rows of a CTA
constexpr int PC_SUB = 16;    // columns of a sub-block
constexpr int PC_MAXCL = 8;   // clusters of a panel (a cluster of 16 SMs per GPC)
constexpr int PC_WARPS = PC_T / 32;
constexpr size_t PC_SMEM_LIMIT = 224 * 1024;  // beside about 2 KB of static shared memory

// bytes of a candidate message: 16 entries, key and row, the reciprocal
constexpr size_t panel_message_bytes(size_t entry) { return PC_SUB * entry + 32; }
// shared memory of a CTA with `chunk` rows of nb columns in a cluster of cs CTAs
constexpr size_t panel_cluster_smem(size_t entry, int chunk, int nb, int cs) {
    return (2 * cs + PC_MAXCL) * panel_message_bytes(entry) + 2 * PC_WARPS * PC_SUB * entry +
           (size_t)PC_SUB * nb * entry + (size_t)chunk * (nb + 1) * entry;
}

struct PanelShape {
    int cs = 0, ncl = 0, chunk = 0;  // CTAs of a cluster, clusters, rows of a CTA; cs 0: the panel does not fit
};

// The cluster panel of `rows` rows and nb columns. least_rows 0: about 64 rows a CTA while one cluster holds
// them (measured per column at 24, 48, 64 and 96 rows: 1.22, 1.19, 1.19, 1.21 us at 240 rows FP64; 1.23,
// 1.22, 1.22, 1.25 at 1920 FP32): fewer rows only add messages, more rows lengthen the rank-16 update. Beyond
// one cluster about 128 rows a CTA: every further cluster adds readers to the global exchange (12288 FP32:
// 1.87 us at 96 and 128 rows, 1.94 at 160, 1.96 at 192), so the first cluster panels of 24576 rows, which
// need all 7 clusters, cost 2.7 us a column. least_rows: so many rows a CTA in either case, as far as they
// fit, for panels that share the chip.
inline PanelShape panel_cluster_shape(size_t entry, int rows, int nb, int least_rows, int most_clusters) {
    PanelShape s;
    if (most_clusters < 1) return s;
    const int one = least_rows > 0 ? least_rows : 64, several = least_rows > 0 ? least_rows : 128;
    int cs = 1, ncl = 1, chunk = 0;
    while (cs < 16 && cs * one < rows) cs *= 2;
    auto fits = [&]() {
        chunk = (rows + cs * ncl - 1) / (cs * ncl);
        return chunk <= PC_T && panel_cluster_smem(entry, chunk, nb, cs) <= PC_SMEM_LIMIT;
    };
    while (cs < 16 && !fits()) cs *= 2;
    if (!fits()) {
        ncl = std::max(1, std::min(most_clusters, (rows + 16 * several - 1) / (16 * several)));
        while (!fits())
            if (++ncl > most_clusters) return s;
    }
    s.cs = cs;
    s.ncl = ncl;
    s.chunk = chunk;
    return s;
}

}  // namespace tcu
