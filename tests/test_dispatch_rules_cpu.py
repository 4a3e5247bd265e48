"""Which of two kernels with the same result a call takes, by its sizes alone (csrc/dispatch_rules.h, through b200_rule_query, no GPU):
both sides of every line, at sizes where both kernels were timed."""
import ctypes as C

import pytest

from kubeai_b200._lib import lib

PICKED_ALONE, KEY_LANES, STREAM, CLUSTER, SEGMENTS, ROW_REGISTERS, ROW_BLOCKS, SINGLE_STEP, LATENT_ROWS = range(9)


def rule(which, *v):
    return lib().b200_rule_query(which, (C.c_int32 * len(v))(*v), len(v))


def test_unknown_rules_are_refused():
    assert rule(99, 1) < 0 and rule(PICKED_ALONE, 1, 2) < 0 and lib().b200_rule_query(PICKED_ALONE, None, 4) < 0


# pairs, N, K: experts of 2048 and of 4096, gate and up side by side
@pytest.mark.parametrize("rows,N,K,alone", [(2, 4096, 2048, 0), (16, 2048, 2048, 0), (24, 2048, 2048, 1), (16, 4096, 2048, 1), (2, 8192, 4096, 0), (4, 8192, 4096, 1),
                                            (32, 8192, 4096, 1), (64, 8192, 4096, 1), (64, 64, 64, 0)])
def test_large_streams_of_picked_rows_run_behind_their_predecessor(rows, N, K, alone):
    """Overlapping a product that holds most of an SM as shared memory, 64 pairs of 8192 x 4096 took 5335 us a step against 4222."""
    assert rule(PICKED_ALONE, rows, N, K, 2) == alone


# tokens, heads, width, keys, cap
@pytest.mark.parametrize("tokens,heads,width,keys,cap,lanes", [
    # few tokens: by width and the length of the chain
    (1, 16, 128, 16, 0, 1), (1, 16, 128, 16000, 0, 1), (1, 16, 128, 8000, 1, 1), (4, 16, 72, 2000, 0, 1), (1, 16, 72, 8000, 0, 0), (1, 16, 96, 1000, 1, 1), (4, 16, 96, 2000, 1, 0),
    (16, 16, 64, 500, 0, 1), (1, 2, 64, 2000, 0, 0), (1, 64, 64, 8000, 0, 0), (16, 6, 40, 4000, 0, 0), (4, 8, 8, 30, 0, 1), (1, 8, 8, 300, 0, 0), (16, 8, 8, 4000, 0, 0),
    # many tokens: by width, cap and the keys there are
    (100, 16, 128, 10, 0, 1), (64, 32, 128, 10, 0, 0), (100, 32, 128, 10, 0, 0), (384, 32, 128, 12, 0, 0), (112, 32, 128, 40, 0, 1), (128, 16, 128, 1000, 0, 1), (100, 32, 128, 10, 1, 0), (112, 32, 128, 40, 1, 0),
    (240, 16, 128, 1200, 1, 1), (128, 16, 72, 20, 0, 0), (128, 16, 72, 250, 0, 1), (240, 8, 64, 1200, 1, 0), (384, 8, 32, 24, 0, 0), (4096, 4, 8, 512, 0, 0)])
def test_sixteen_lanes_hold_a_key_where_that_is_faster(tokens, heads, width, keys, cap, lanes):
    """Everywhere, they took 294 us against 124 for 8 heads of 8 over 16000 keys, and 56 against 36 for 100 tokens of up to 10 keys, 32 capped heads of 128."""
    assert rule(KEY_LANES, tokens, heads, width, keys, cap) == lanes


@pytest.mark.parametrize("T,N,K,pairs,pays", [(48, 2048, 8192, 0, 1), (40, 1024, 14336, 0, 0), (48, 3168, 14336, 0, 0), (40, 4096, 14336, 0, 1), (48, 4096, 14336, 0, 1), (32, 2048, 14336, 0, 1),
                                               (32, 1024, 28672, 0, 0), (32, 2048, 28672, 0, 1), (16, 1024, 28672, 0, 1), (48, 1024, 28672, 0, 0), (8, 576, 28672, 0, 1),
                                               (24, 7168, 16384, 1, 1), (32, 7168, 16384, 1, 0), (32, 7168, 8192, 1, 1), (8, 28672, 4096, 1, 1)])
def test_passes_over_the_weights_end_where_a_long_k_makes_x_the_larger_part(T, N, K, pairs, pays):
    """Lines drawn by T and N alone sent 40 rows of 1024 x 28672 through them: 49 us against 33 in whole tiles."""
    assert rule(STREAM, T, N, K, pairs) == pays


@pytest.mark.parametrize("T,N,K,pays", [(100, 2048, 2048, 1), (256, 2112, 8192, 1), (100, 1024, 14336, 1), (129, 1024, 14336, 0), (100, 2048, 28672, 0), (64, 3072, 4096, 1), (64, 3072, 8192, 0),
                                         (128, 3168, 648, 1)])
def test_clusters_end_there_too(T, N, K, pays):
    """129 rows of 2048 x 28672: 72 us in clusters, 53 in whole tiles."""
    assert rule(CLUSTER, T, N, K) == pays


# heads, column blocks, state rows, sequences, tokens of each
@pytest.mark.parametrize("heads,blocks,dim,nseq,each,cut", [
    (8, 1, 128, 1, 4096, 1), (8, 1, 128, 6, 682, 1), (16, 1, 128, 4, 1024, 1), (32, 1, 128, 4, 512, 0), (32, 1, 128, 6, 682, 0), (32, 1, 128, 4, 1024, 1),
    (64, 1, 128, 1, 512, 1), (64, 1, 128, 1, 4096, 1), (64, 1, 128, 2, 512, 0), (64, 1, 128, 3, 1365, 1), (64, 1, 128, 4, 512, 0), (64, 1, 128, 4, 1024, 0),
    (128, 1, 128, 1, 1024, 1), (128, 1, 128, 2, 512, 0), (128, 1, 128, 2, 2048, 0), (128, 1, 128, 4, 1024, 0), (256, 1, 128, 1, 512, 0), (256, 1, 128, 1, 4096, 0),
    (256, 1, 128, 3, 1365, 0), (32, 2, 128, 4, 512, 0), (64, 4, 64, 1, 512, 0), (64, 1, 16, 5, 820, 0), (64, 1, 16, 1, 4096, 1), (8, 1, 128, 7, 1024, 0), (8, 1, 128, 4, 500, 0)])
def test_sequences_are_cut_where_their_chains_leave_the_device_idle(heads, blocks, dim, nseq, each, cut):
    """By sequences and tokens alone, four of 512 tokens with 64 heads were cut: 171 us against 114 in chains."""
    for longest in (each, 0):
        assert rule(SEGMENTS, nseq * each, nseq, longest, heads, blocks, dim, 444 if dim <= 32 else 296, 148) == cut


@pytest.mark.parametrize("heads,dim,nseq,each,cut", [(64, 128, 6, 682, 0), (64, 128, 2, 1024, 1), (128, 64, 2, 2048, 0), (256, 64, 1, 4096, 0), (128, 64, 3, 1365, 1),
                                                     (64, 32, 4, 1024, 0), (128, 32, 2, 2048, 0), (64, 32, 1, 1024, 1), (256, 32, 1, 4096, 0)])
def test_chains_whose_tiles_come_in_ahead_stay_whole_longer(heads, dim, nseq, each, cut):
    """128 heads, 64 state rows, two sequences of 2048: 253 us in segments, 303 in chains that waited for each chunk's tiles, 211 since."""
    assert rule(SEGMENTS, nseq * each, nseq, each, heads, 1, dim, 444 if dim <= 32 else 296, 148) == cut


def test_a_chain_is_as_long_as_its_longest_sequence():
    assert rule(SEGMENTS, 4095, 3, 2275, 64, 1, 128, 296, 148) == 1 and rule(SEGMENTS, 4096, 4, 3000, 64, 1, 128, 296, 148) == 1
    assert rule(SEGMENTS, 4100, 4, 2000, 128, 1, 128, 296, 148) == 1 and rule(SEGMENTS, 2300, 2, 2000, 256, 1, 128, 296, 148) == 0
    assert rule(SEGMENTS, 4000, 6, 1200, 64, 1, 128, 296, 148) == 1 and rule(SEGMENTS, 4000, 6, 1200, 128, 1, 128, 296, 148) == 0


@pytest.mark.parametrize("pieces,rows,held", [(1, 4096, 1), (2, 4096, 1), (3, 444, 1), (3, 445, 0), (4, 1, 1), (4, 148, 1), (4, 4000, 0), (5, 1, 0)])
def test_wide_rows_stay_in_registers_in_steps_and_not_in_prompts(pieces, rows, held):
    """4000 rows of 4096 held in registers took 232 us in nine launches, 196 read again behind each sum."""
    assert rule(ROW_REGISTERS, pieces, rows, 148) == held


@pytest.mark.parametrize("rows,heads,N,K,fp32,blocks", [(64, 16, 512, 128, 0, 1), (128, 16, 512, 128, 0, 0), (32, 32, 512, 128, 0, 1), (100, 32, 512, 128, 0, 0), (128, 64, 512, 128, 0, 0),
                                                         (128, 4, 512, 128, 0, 1), (128, 64, 256, 64, 0, 0), (100, 32, 256, 64, 0, 0), (64, 16, 256, 64, 0, 1), (100, 16, 128, 512, 1, 1), (64, 64, 128, 512, 1, 1), (128, 64, 128, 512, 1, 0),
                                                         (128, 64, 64, 256, 1, 1)])
def test_products_per_head_in_blocks_of_rows_while_their_reads_of_the_weights_are_few(rows, heads, N, K, fp32, blocks):
    """Whatever the heads, 100 rows of 32 heads, 128 to 512 columns, took 18.8 us in blocks against 14.9 in tiles."""
    assert rule(ROW_BLOCKS, rows, heads, N, K, fp32) == blocks


@pytest.mark.parametrize("units,dim,vdim,delta,step", [(2048, 128, 128, 0, 1), (2048, 128, 4, 0, 1), (2048, 256, 4, 0, 0), (2048, 256, 32, 0, 1), (2048, 64, 4, 0, 1), (64, 256, 4, 0, 1),
                                                        (2048, 16, 256, 1, 0), (2048, 16, 64, 1, 1), (512, 32, 96, 1, 0), (2048, 64, 256, 1, 1), (512, 128, 16, 1, 0), (512, 128, 32, 1, 1),
                                                        (2048, 256, 8, 1, 0), (2048, 256, 64, 1, 1), (64, 256, 4, 1, 1), (37, 16, 256, 1, 1), (38, 16, 256, 1, 0)])
def test_single_tokens_pass_over_states_that_fill_the_pass(units, dim, vdim, delta, step):
    """Whatever the state, 16 heads of 16 x 256, 128 sequences of the delta rule, took 46.6 us in the pass against 34.2 in the scan."""
    assert rule(SINGLE_STEP, units, dim, vdim, delta, 148) == step


@pytest.mark.parametrize("rank,tokens,held", [(1024, 8, 1), (1024, 4096, 1), (1025, 8, 0), (2048, 4096, 0), (512, 8, 1), (512, 2048, 1), (512, 4096, 0), (128, 512, 1), (128, 4096, 0),
                                               (0, 8, 1), (0, 4096, 0)])
def test_latent_rows_stay_in_registers_where_there_is_room(rank, tokens, held):
    """A kernel with room for 1024 numbers in registers whatever the row: 4096 tokens of 2048 in two layers 73 us against 60."""
    assert rule(LATENT_ROWS, rank, tokens) == held


TILES, TILE_ROWS, TILE_PARTS = 9, 10, 11


@pytest.mark.parametrize("T,N,K,ahead", [(24, 1024, 14336, 0), (28, 1024, 14336, 1), (32, 3168, 14336, 0), (32, 2048, 8192, 0), (40, 2048, 4096, 0), (40, 1024, 8192, 1), (48, 3072, 8192, 1), (40, 4096, 8192, 0),
                                         (40, 2048, 14336, 1), (48, 4096, 14336, 0), (64, 2048, 2048, 0), (128, 2048, 4096, 0), (64, 2048, 8192, 1), (64, 3072, 1024, 1), (129, 1024, 2048, 1), (256, 2048, 2048, 1)])
def test_tiles_chosen_for_the_call_against_the_products_of_few_rows(T, N, K, ahead):
    """40 rows of 1024 x 14336 take 24 us as a pass over the weights, 20 in clusters and 15 in tiles; 64 of 2048 x 2048 8.0 in clusters and 9.5 in tiles."""
    assert rule(TILES, T, N, K) == ahead


@pytest.mark.parametrize("rows,N,K,tile,parts", [(1999, 4096, 14336, 224, 1), (2048, 4096, 14336, 240, 1), (3001, 2048, 2048, 176, 1), (4096, 2048, 8192, 240, 1), (256, 4096, 14336, 128, 2),
                                                 (128, 4096, 4096, 64, 1), (64, 512, 4096, 32, 6), (300, 28672, 4096, 160, 1), (1, 256, 64, 16, 1)])
def test_rows_of_a_tile_and_pieces_of_k(rows, N, K, tile, parts):
    """2048 rows of 4096 x 14336 in tiles of 256 rows are two rounds of 74 pairs with 20 of them idle: 190 us, 178 in tiles of 240."""
    assert (rule(TILE_ROWS, rows, N, K, 74, 1), rule(TILE_PARTS, rows, N, K, 74, 1)) == (tile, parts)


def test_every_choice_of_tiles_can_be_launched():
    """Whole steps of 16 rows, at most 256, and a part of K for every pair at most once."""
    for rows in (1, 15, 16, 17, 31, 33, 100, 128, 129, 255, 256, 257, 500, 511, 1000, 1025, 2049, 4096):
        for N in (8, 256, 520, 2048, 6144, 28672):
            for K in (8, 64, 520, 4096, 14336):
                for pairs in (1, 66, 74):
                    t, p = rule(TILE_ROWS, rows, N, K, pairs, 1), rule(TILE_PARTS, rows, N, K, pairs, 1)
                    tiles = -(-N // 256) * -(-rows // t)
                    assert 16 <= t <= 256 and t % 16 == 0 and p >= 1 and p <= -(-K // 64)
                    assert p == 1 or tiles * p <= pairs
                    assert rule(TILE_PARTS, rows, N, K, pairs, 0) == 1


@pytest.mark.parametrize("ctas,lens,ahead", [
    (32, [63, 191, 319, 447, 575, 703, 831, 959], 1), (64, [63, 191, 319, 447, 575, 703, 831, 959], 0), (32, [1000] * 4 + [500], 1), (32, [777] * 5, 0), (32, [200] * 8, 0),
    (64, [100, 200, 100, 2000, 300, 80], 1), (8, [1000, 1000], 1), (74, [1000, 1000], 1), (80, [1000, 1000], 0), (148, [1000, 1000], 0), (128, [100, 3000], 1), (32, [64], 0),
    (32, [65], 1), (1, [1], 0), (8, [17] * 40, 0), (8, [64] * 40, 0), (4, [64] * 8, 0), (4, [65] * 8, 1)])
def test_delta_scores_come_ahead_where_the_longest_chain_outlasts_the_work(ctas, lens, ahead):
    """16 heads, 5 sequences of 777 tokens: 217 us two CTAs to an SM, 244 with more warps a CTA and one to an SM; 63 to 959 tokens in 8 sequences: 229 and 162."""
    assert rule(12, ctas, len(lens), sum(lens), max(lens), 148) == ahead
    assert rule(12, ctas, len(lens), sum(lens), 0, 148) == (sum(lens) > 64 and ctas * len(lens) <= 148)


GATE_UP, STEP_TILES = 13, 14


@pytest.mark.parametrize("N,K,tiles", [(28672, 4096, 1), (14336, 4096, 1), (18944, 8192, 1), (19456, 8192, 0), (19456, 4096, 0), (19456, 2048, 1), (20480, 5120, 0), (22016, 8192, 0), (22016, 4096, 1),
                                       (24576, 8192, 1), (37888, 8192, 1), (38912, 8192, 1), (57344, 8192, 1), (256, 64, 1)])
def test_few_gate_and_up_tiles_left_for_a_second_round_stay_with_the_pairs(N, K, tiles):
    """19456 x 8192 is 76 tiles on 74 pairs, 64 rows: 66 us in two rounds, 61 where the pairs share out the steps of K."""
    assert rule(GATE_UP, N, K, 74) == tiles


@pytest.mark.parametrize("tokens,hidden,form", [(9, 1024, 1), (48, 1024, 1), (49, 1024, 0), (64, 1024, 0), (65, 1024, 2), (49, 2048, 1), (64, 2048, 1), (65, 4096, 2), (128, 4096, 2)])
def test_projections_of_a_step(tokens, hidden, form):
    assert rule(STEP_TILES, tokens, hidden) == form


@pytest.mark.parametrize("rows,N,K,tile", [(700, 11008, 8192, 240), (700, 11008, 14336, 240), (1000, 19456, 14336, 256), (600, 14336, 1024, 128), (300, 28672, 14336, 112), (700, 2048, 8192, 112)])
def test_of_choices_that_are_even_the_fewest_tiles(rows, N, K, tile):
    """700 rows of 11008 x 14336: 129 tiles of 240 rows 160 us, 215 of 144 rows 178, although the busiest pair has fewer rows then."""
    assert rule(TILE_ROWS, rows, N, K, 74, 1) == tile


def test_clusters_have_whole_tiles_to_beat_only_in_short_products():
    """What tiles_ahead leaves the clusters (49 rows on, where the passes end) is all theirs; cluster_pays draws its own lines for outputs that are no whole 16-byte pieces."""
    for T in range(49, 257):
        for N in (8, 1024, 2112, 2120, 3168, 4096):
            for K in (512, 2048, 6144, 6208, 8192, 14336):
                if not rule(TILES, T, N, K):
                    assert T <= 128 and N <= 2112 and K <= 6144 and rule(CLUSTER, T, N, K) == 1
