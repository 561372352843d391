// Host rules of csrc/kv_plan.h: what they choose is the same for every length of one 640-position bucket, so the number of query tokens
// cannot change it. With arguments n, T, pos_lo, pos_hi, layers: prints the length of a range's pieces.
#include <cstdio>
#include <cstdlib>

#include "kv_plan.h"

using namespace mkkv;

static AttnJob job(int L, int T, int lo, int hi) {
    AttnJob j{};
    j.n = L - T;
    j.T = T;
    attn_dims(L, j.nch, j.cs);
    j.cpi = chunks_per_item(j.cs);
    j.pos_lo = lo;
    j.pos_hi = std::min(L, hi);
    j.c_lo = lo / j.cs;
    j.nch = (j.pos_hi + j.cs - 1) / j.cs - j.c_lo;
    return j;
}

// which mode a call takes: one answer per bucket, for whole contexts and for ranges; one layer leaves the one launch once
static int modes() {
    int bad = 0;
    for (int nlayers : {1, 2, 3, 4, 8, 16}) {
        int switches = 0, before = -1;
        for (int bucket = 1; bucket <= 262144 / ATT_BUCKET; bucket += bucket < 40 ? 1 : 7) {
            const int top = bucket * ATT_BUCKET, starts[3] = {0, top / 3 / ATP * ATP, (top - 1) / ATT_BUCKET * ATT_BUCKET};
            for (int lo : starts) {
                const int ends[3] = {1 << 30, std::max(lo + ATP, top - 5 * ATP), std::max(lo + ATP, top / 2 / ATP * ATP)};
                for (int hi : ends) {
                    int first = -1;
                    for (int L = top - ATT_BUCKET + 1; L <= top; L += top - L < 10 ? 1 : 9) {
                        if (std::min(L, hi) <= lo) continue;
                        for (int T : {1, 8}) {
                            if (L < T) continue;
                            const int m = items_mode(nlayers, job(L, T, lo, hi), 148);
                            if (first >= 0 && m != first) bad++ < 5 ? std::printf("%d layers, length %d, range %d .. %d: %d\n", nlayers, L, lo, hi, m) : 0;
                            first = m;
                        }
                    }
                    if (lo == 0 && hi == 1 << 30) switches += before >= 0 && first != before, before = first;
                }
            }
        }
        if (nlayers == 1 && switches != 1) bad++, std::printf("one layer: %d switches\n", switches);
    }
    return bad;
}

// a range's pieces: one length per bucket, whole groups, no longer than a chunk, no more of them than the partials' scratch holds
static int pieces() {
    int bad = 0, cut = 0;
    for (int layers : {1, 8, 16})
        for (int bucket = 1; bucket <= 262144 / ATT_BUCKET; bucket += bucket < 70 ? 3 : 13)
            for (int world : {1, 2, 3, 8})
                for (int rank = 0; rank < world; rank++) {
                    const int top = bucket * ATT_BUCKET, share = (top + 64 + world - 1) / world / ATP * ATP + ATP, lo = rank * share, hi = lo + share;
                    int first = -1;
                    for (int L = top - ATT_BUCKET + 1; L <= top; L += top - L < 10 ? 1 : 61)
                        for (int T : {1, 8}) {
                            if (L < T || std::min(L, hi) <= lo) continue;
                            AttnJob j = job(L, T, lo, hi);
                            const int p = range_piece(layers, j);
                            const int n = (j.pos_hi + p - 1) / p - lo / p;
                            const bool ok = (first < 0 || p == first) && p <= j.cs && (p == j.cs || p % GROUP == 0) && n <= ATT_NCH && (bucket > 63 || p == j.cs);
                            if (!ok) bad++ < 5 ? std::printf("%d layers, length %d, range %d .. %d: pieces of %d, chunks of %d\n", layers, L, lo, hi, p, j.cs) : 0;
                            first = p;
                            cut += p != j.cs;
                        }
                }
    if (!cut) bad++, std::printf("no range was cut\n");
    return bad;
}

// 2,000 decode steps of 1 to 8 tokens, then another sequence's: the rules are evaluated once per bucket, with the same answers
static int memo() {
    PlanMemo mode, piece;
    int runs = 0, bad = 0, T = 1;
    for (int n : {60000, 90000})
        for (int i = 0, at = n; i < 2000; i++, at += T) {
            T = att_cap_T(at, 1 + i % 8);
            const AttnJob j = job(at + T, T, 32768, 65536);
            const std::array<int, 4> key = {16, j.cs, j.pos_lo, plan_end(j)};
            bad += piece.get(key, [&] { return runs++, range_piece(16, j); }) != range_piece(16, j);
            bad += mode.get(key, [&] { return runs++, (int) items_mode(16, j, 148); }) != (int) items_mode(16, j, 148);
        }
    const int buckets = 2 * (2000 * 9 / 2 / ATT_BUCKET + 2);
    if (bad || runs > 2 * buckets) std::printf("%d answers differ, %d evaluations\n", bad, runs);
    return bad + (runs > 2 * buckets);
}

int main(int argc, char ** argv) {
    if (argc == 6) {
        const int n = atoi(argv[1]), T = atoi(argv[2]);
        std::printf("%d\n", range_piece(atoi(argv[5]), job(n + T, T, atoi(argv[3]), atoi(argv[4]))));
        return 0;
    }
    return modes() + pieces() + memo() != 0;
}
