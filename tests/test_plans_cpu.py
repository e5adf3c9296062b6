"""The rules that pick a kernel and a tile for a product (plan_chain), asked through a small program that links the library: host code,
no device needed."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "zoph_rnn_b200")
BF16, TF32, TF32X3, F16X2 = range(4)
STORE, LSTM = range(2)

PROBE = r"""
#include <chrono>
#include <cstdio>
#include "skinny_gemm.cuh"
#include "tc_chain.cuh"
#include "tc_vocab.cuh"
// lines of "mode epi rows nsrc kb n_early columns beside cells H" -> "BN split nb microseconds skinny"; one call takes that long at least of
// three; skinny: the warp-level kernel's estimate is the shorter one
int main(int argc, char**) {
  if (argc > 1) {  // lines of "mode kb columns words" -> "column tiles, columns of a tile, log-sum-exp in tiles of one CTA"
    int mode, kb, M, N;
    while (std::scanf("%d %d %d %d", &mode, &kb, &M, &N) == 4) {
      const zrnn::VocabTiles t = zrnn::vocab_pair_tiles(M, N);
      std::printf("%d %d %d\n", t.n_ct, t.nb, (int)zrnn::vocab_lse_single(mode, kb, M, N));
    }
    return 0;
  }
  int mode, epi, rows, nsrc, kb, early, M, beside, cells, H;
  while (std::scanf("%d %d %d %d %d %d %d %d %d %d", &mode, &epi, &rows, &nsrc, &kb, &early, &M, &beside, &cells, &H) == 10) {
    zrnn::ChainPlan p;
    double best = 1e30;
    for (int i = 0; i < 3; ++i) {
      const auto t0 = std::chrono::steady_clock::now();
      p = zrnn::plan_chain(mode, epi, rows, cells, nsrc, kb, early, M, beside != 0);
      const double us = std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count();
      if (us < best) best = us;
    }
    const int sk = epi == zrnn::TC_EPI_LSTM ? zrnn::SK_EPI_LSTM : zrnn::SK_EPI_STORE;
    const bool skinny = M <= 64 && (mode == zrnn::TC_BF16 || mode == zrnn::TC_F16X2) &&
                        (zrnn::skinny_us(mode == zrnn::TC_BF16 ? zrnn::SK_BF16 : zrnn::SK_F16X2, sk, rows, nsrc * H, M, cells, early > 0 && !beside) < p.us ||
                         (mode == zrnn::TC_F16X2 && zrnn::skinny_more_exact(sk, rows, cells, nsrc, H, early, M)));
    std::printf("%d %d %d %g %d\n", p.BN, p.split, p.nb, best, (int)skinny);
  }
}
"""


def kblocks(mode, H):
    per = 64 if mode in (BF16, F16X2) else 32
    return (H + per - 1) // per


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    from zoph_rnn_b200 import build
    lib = build.build()
    d = tmp_path_factory.mktemp("plans")
    src, exe = str(d / "probe.cpp"), str(d / "probe")
    with open(src, "w") as f:
        f.write(PROBE)
    cuda = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-I" + os.path.join(cuda, "include"), "-I" + os.path.join(PKG, "csrc"), src,
                           "-o", exe, lib, "-Wl,-rpath," + PKG])

    def ask(questions, vocab=False):
        if vocab:
            out = subprocess.run([exe, "vocab"], input="".join("%d %d %d %d\n" % q for q in questions), stdout=subprocess.PIPE, text=True, check=True)
            return [tuple(int(x) for x in line.split()) for line in out.stdout.splitlines()]
        lines = "".join("%d %d %d %d %d %d %d %d %d %d\n" % (q if len(q) == 10 else q + (1, 1)) for q in questions)
        out = subprocess.run([exe], input=lines, stdout=subprocess.PIPE, text=True, check=True)
        rows = [(int(a), int(b), int(c), float(t), int(k)) for a, b, c, t, k in (line.split() for line in out.stdout.splitlines())]
        assert len(rows) == len(questions)
        return rows
    return ask


def test_single_pass_products_are_summed_over_two_parts_at_most(plans):
    """A product of the single-pass modes is rounded to 10 or 7 bits at its end, so another order of its sums turns some of its results by a
    unit there: four parts of the K axis gave a bf16 scoring pass other values for 0.4 % of its time, and are for the split modes."""
    q = [(mode, STORE, rows, nsrc, kblocks(mode, H), 0, M, beside) for mode in (BF16, TF32) for H in (256, 500, 1000, 1024, 2048)
         for rows, nsrc in ((H, 2), (2 * H, 1)) for M in (1, 12, 64, 100, 128, 200, 256, 400, 768) for beside in (0, 1)]
    assert max(p[1] for p in plans(q)) == 2
    assert any(p[1] == 4 for p in plans([(F16X2, STORE, 1000, 2, 16, 0, M, 0) for M in (64, 128)]))


def waves(M, rows, width, split=1):
    return -(-(-(-M // 128) * -(-rows // width) * split) // 148)


def test_one_accumulator_over_the_whole_k_axis_only_where_it_halves_the_waves(plans):
    """Tiles of more than 160 columns on pairs of CTAs give each split-mode product one truncating accumulator for the whole K axis, several
    times as far from float64 as rounds.  Never in 3xTF32; in the fp16 split where, and only where, tiles of 256 weight rows on single CTAs, which
    had such an accumulator too, took so much less than tiles of 128 rows, and of 64 rows that have early sources, that they were chosen:
    1000 units at 768 columns, not at 1500, and not where two of three sources are early."""
    q = [(mode, epi, (4 if epi == LSTM else 2 if nsrc == 1 else 1) * H, nsrc, kblocks(mode, H), early, M, 0) for mode in (TF32X3, F16X2) for epi in (STORE, LSTM)
         for H in (256, 320, 400, 500, 512, 640, 768, 900, 1000, 1024, 1536, 2048) for nsrc in (1, 2, 3) for early in range(nsrc) for M in range(257, 4100, 31)]
    seen = set()
    for (mode, epi, rows, nsrc, kb, early, M, _), (_, _, nb, _, _) in zip(q, plans(q)):
        if nb > 160:
            w = waves(M, rows, 256)
            assert mode == F16X2 and waves(M, rows, 128) > 1.6 * w, (mode, epi, rows, nsrc, M, nb)
            assert (nsrc - early / 2) * min(waves(M, rows, 64), waves(M, rows, 64, 2) / 2) > 2 * nsrc * w, (mode, epi, rows, nsrc, early, M, nb)
            seen.add((rows, early))
    assert (4000, 0) in seen and (4000, 1) in seen  # (the rule is reached)
    cell = [(F16X2, LSTM, 4000, 2, 16, 0, M, 0) for M in (600, 768, 1024, 1440, 1500, 1640)]
    nb = [p[2] for p in plans(cell)]
    assert nb[1] > 160 and nb[2] > 160 and all(n <= 160 for n in nb[3:]), nb
    feed = [(F16X2, LSTM, 4 * H, 3, kblocks(F16X2, H), 2, M, 0) for H, M in ((1000, 700), (1000, 890), (768, 1000), (900, 700), (2048, 350))]
    assert all(p[2] <= 160 for p in plans(feed))


def test_very_many_columns_are_planned_in_no_time_and_fit_a_grid(plans):
    """A plan is made at every launch, so it must not look at every way to cut millions of columns into tiles; and the column tiles of pairs of
    CTAs are the second axis of a grid, which ends at 65535: beyond, the tiles of single CTAs, whose columns are the first axis, take them."""
    q = [(mode, STORE, rows, 1, kb, 0, M, 0) for mode in (BF16, TF32, TF32X3, F16X2) for rows in (64, 256, 2000) for kb in (1, 4, 16)
         for M in (70000, 1 << 20, 10_500_000, 17_000_000, 30_000_000)]
    for (mode, _, rows, _, _, _, M, _), (BN, split, nb, us, _) in zip(q, plans(q)):
        assert nb == 0 or -(-M // nb) <= 65535, (mode, rows, M, nb)
        assert us < 20, (M, us)


# kind of link (epilogue, weight rows per H, sources, early ones), cells in the launch, mode, H, columns -> the kernels (warp-level: "skinny", else
# tile rows / CTAs per tile) within 3 % of the best pass; with the next best one a pass took 2 - 28 % longer
MEASURED = [("cell", 1, BF16, 320, 1, "skinny"), ("cell", 1, BF16, 320, 8, "skinny"), ("cell", 1, BF16, 320, 16, "skinny"), ("cell", 1, BF16, 504, 16, "skinny"),
            ("cell", 1, BF16, 400, 24, "skinny"), ("cell", 1, BF16, 400, 128, "32/2"), ("cell", 1, BF16, 1000, 128, "64/2"), ("cell", 1, F16X2, 256, 100, "32/2"),
            ("cell", 1, F16X2, 504, 64, "64/2"), ("cell", 1, F16X2, 256, 200, "32/1 64/2"), ("cell", 1, F16X2, 1000, 1, "skinny"), ("cell", 1, F16X2, 1000, 16, "skinny"),
            ("cell", 1, TF32X3, 504, 4, "64/2"), ("stack", 2, BF16, 1000, 1, "skinny"), ("stack", 2, BF16, 1000, 8, "skinny"), ("stack", 4, BF16, 256, 40, "32/1"),
            ("stack", 2, F16X2, 1000, 12, "skinny"), ("stack", 2, F16X2, 1000, 16, "skinny"), ("stack", 3, F16X2, 640, 12, "skinny"), ("stack", 3, F16X2, 640, 16, "skinny"),
            ("stack", 4, F16X2, 400, 24, "skinny"), ("stack", 4, F16X2, 640, 32, "64/1 128/1"), ("stack", 3, F16X2, 1000, 24, "64/1 128/1"), ("stack", 4, F16X2, 1000, 56, "128/1"),
            ("stack", 4, F16X2, 1000, 128, "128/1"), ("stack", 4, BF16, 1000, 128, "128/1"), ("projection", 1, F16X2, 400, 100, "32/4 32/2"), ("projection", 1, F16X2, 504, 80, "32/4 32/2")]


def test_links_take_the_kernel_that_was_measured_to_be_faster(plans):
    """Shapes at which the refitted rule of the links had left the faster kernel, and some at which it had not: passes of 10 + 10 steps, 1000 words."""
    kinds = {"cell": (LSTM, 4, 2, 1), "stack": (LSTM, 4, 2, 0), "projection": (STORE, 2, 1, 0)}
    q = []
    for kind, cells, mode, H, M, _ in MEASURED:
        epi, per, nsrc, early = kinds[kind]
        q.append((mode, epi, per * H, nsrc, kblocks(mode, H), early, M, 0, cells, H))
    got = ["skinny" if sk else "%d/%d" % (BN, split) for BN, split, _, _, sk in plans(q)]
    assert [(m, g) for m, g in zip(MEASURED, got) if g not in m[5].split()] == []


def test_vocabulary_tiles_cover_the_columns(plans):
    """What the pair kernel asks of its tiles, for all numbers of columns and some large ones: a multiple of 32 columns, none of the tiles empty."""
    q = [(F16X2, 16, M, N) for N in (1, 700, 3000, 50000, 1 << 20) for M in list(range(65, 1500, 7)) + [16384, 70001, 1 << 20]]
    for (_, _, M, N), (n_ct, nb, _) in zip(q, plans(q, vocab=True)):
        assert 32 <= nb <= 256 and nb % 32 == 0 and n_ct * nb >= M > (n_ct - 1) * nb, (M, N, n_ct, nb)


# mode, K, words, columns -> columns of a tile (0: any), log-sum-exp in tiles of one CTA; what the other choice takes is 9 - 45 % longer
MEASURED_VOCAB = [(F16X2, 1000, 700, 1200, 64, False), (F16X2, 504, 700, 500, 32, False), (TF32X3, 1000, 700, 500, 32, False), (F16X2, 504, 3000, 768, 0, True),
                  (F16X2, 504, 3000, 500, 0, True), (TF32X3, 256, 3000, 768, 0, True), (F16X2, 504, 10000, 500, 0, True), (F16X2, 504, 10000, 100, 0, True),
                  (F16X2, 1000, 40000, 768, 256, False), (F16X2, 1000, 50000, 6400, 0, False), (F16X2, 1000, 50000, 160, 160, False), (BF16, 2048, 200000, 16384, 256, False),
                  (BF16, 1000, 50000, 6400, 0, True), (F16X2, 100, 10000, 280, 0, True)]


def test_vocabulary_projection_takes_the_tiles_that_were_measured_to_be_faster(plans):
    got = plans([(mode, kblocks(mode, K), M, N) for mode, K, N, M, _, _ in MEASURED_VOCAB], vocab=True)
    assert [(m, g) for m, g in zip(MEASURED_VOCAB, got) if (m[4] and g[1] != m[4]) or bool(g[2]) != m[5]] == []


def test_many_columns_take_pairs_of_ctas_only_where_they_are_faster(plans):
    """Every wave of pairs pays its set-up and its end anew, so tiles of 128 x 128 on single CTAs, of which twice as many run at a time, can be
    faster: us per cell, pairs / single CTAs, bf16, 504 units, 2100 columns 18.8 / 16.7, 1000 units, 900 columns 23.9 / 23.4; fp16 split, 504 units, 3000 columns
    61.8 / 47.3; but 1000 units, 768 columns in bf16 19.8 / 22.6."""
    q = [(BF16, 504, 2100, False), (BF16, 1000, 900, False), (BF16, 1000, 1024, False), (F16X2, 504, 3000, False), (F16X2, 1000, 1300, True), (BF16, 1000, 768, True), (F16X2, 2048, 600, True)]
    got = plans([(mode, LSTM, 4 * H, 2, kblocks(mode, H), 0, M, 0) for mode, H, M, _ in q])
    assert [(a, p[2]) for a, p in zip(q, got) if (p[2] > 0) != a[3]] == []


def test_the_more_exact_kernel_keeps_its_shapes(plans):
    """Accumulators of the warp-level kernel absorb fewer products than those of the links, so in the fp16 split the refitted estimates do not take
    shapes from it: the largest numbers of columns at which it was chosen when links were issued by one thread (kind, H -> columns)."""
    kept = [("cell", 500, 32), ("cell", 640, 24), ("cell", 320, 64), ("product", 500, 64), ("product", 768, 64), ("product", 1000, 48), ("product", 1024, 48),
            ("stacked", 640, 64), ("stacked", 1000, 40), ("stacked", 1200, 40)]
    kinds = {"cell": (LSTM, 4, 2, 1), "product": (STORE, 1, 2, 1), "stacked": (STORE, 2, 1, 0)}
    q = [(kinds[k][0], kinds[k][1] * H, kinds[k][2], kinds[k][3], H, M) for k, H, top in kept for M in (1, top // 2, top)]
    got = plans([(F16X2, epi, rows, nsrc, kblocks(F16X2, H), early, M, 0, 1, H) for epi, rows, nsrc, early, H, M in q])
    assert [(a, g) for a, g in zip(q, got) if not g[4]] == []
