"""The mbarrier protocol of the key-loop tcgen05 kernels, checked on the CPU with a discrete-event model
(tests/protocol_model.py): random latencies, random piece shapes, hardware parity semantics, ownership assertions on
every tensor-memory buffer and ring stage.  No GPU run can show the absence of a race; a few hundred random schedules of
the model at least show the protocol has none that depends on who is faster."""
import random

import pytest

from protocol_model import (coarse_selection_kernel, forward_kernel, key_major_kernel, outcome, query_major_kernel, single_shot_backward_kernel,
                            single_shot_forward_kernel)

RUNS = 250


def _pieces(seed):
    rng = random.Random(seed)
    return [rng.randint(1, 25) for _ in range(rng.randint(1, 4))]          # odd and even unit lengths, units of one job


def test_key_major_kernel_protocol_has_no_hazard_or_deadlock():
    """attn_dkv_pooled_loop_tc_kernel, dense form: two producers, one S^T / dP^T warp, one dV / dK warp, four S^T and two dP^T buffers,
    barriers per buffer, epilogue warps."""
    for seed in range(RUNS):
        assert outcome(key_major_kernel, seed, _pieces(seed)) == "ok", seed


def test_query_major_kernel_protocol_has_no_hazard_or_deadlock():
    """attn_dq_pooled_loop_tc_kernel: two producers, one S / dP warp, one dQ warp, two accumulators, epilogue warps."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        assert outcome(query_major_kernel, seed, rng.randint(1, 7), rng.choice([4, 6, 18])) == "ok", seed


@pytest.mark.parametrize("passes", [1, 2])
def test_forward_kernel_protocol_has_no_hazard_or_deadlock(passes):
    """attn_fwd_pooled_loop_tc_kernel with three softmax groups in its one-pass form (with 2 and 8 chunks a tile's first job goes round the groups,
    with 3 and 9 it is always the same group's) and in the two-pass form."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        assert outcome(forward_kernel, seed, rng.randint(1, 6), rng.choice([2, 3, 8, 9]), passes) == "ok", seed


def test_model_catches_the_parity_hazard_of_two_score_threads():
    """The model has teeth: S / dP of even and odd jobs on TWO threads with barriers per BUFFER is the variant that read
    scores before they were written on the GPU.  A softmax group asks for the second completion of a barrier whose first
    completion belongs to the other thread and has not happened yet; the parity test passes.  The model finds it within
    a few schedules, in both kernels."""
    bad_kv = sum(outcome(key_major_kernel, s, _pieces(s), score_threads=2) != "ok" for s in range(60))
    bad_q = sum(outcome(query_major_kernel, s, 4, 6, score_threads=2) != "ok" for s in range(60))
    assert bad_kv > 0 and bad_q > 0


@pytest.mark.parametrize("kernel", ["key_major", "query_major"])
def test_barriers_per_job_number_mod_6_make_two_score_threads_safe(kernel):
    """With sdp_ready / buf_free indexed by the job number mod 6 every barrier has one committing thread and one waiting
    thread or group that meet its phases in order: the two-thread variant is then safe (it ran parity-green with device
    checks on, and no faster than the one-thread form, which is why the kernels keep the simpler one)."""
    for seed in range(RUNS):
        if kernel == "key_major":
            r = outcome(key_major_kernel, seed, _pieces(seed), score_threads=2, score_barriers=6)
        else:
            rng = random.Random(seed)
            r = outcome(query_major_kernel, seed, rng.randint(1, 7), rng.choice([4, 6, 18]), score_threads=2, score_barriers=6)
        assert r == "ok", seed


def _single_shot_case(seed):
    rng = random.Random(seed)
    return rng.randint(0, 9), rng.randint(1, 14), rng.choice([2, 4, 8, 128])       # first tile, tiles of the CTA, tiles per head


def test_single_shot_backward_protocol_has_no_hazard_or_deadlock():
    """attn_bwd_pooled_tc_kernel as built: TMA producer, two MMA-issuing threads (S / dP / dQ; the transposed products) that
    both commit out_ready and mma_done, twelve softmax warps, four drain warps; CTA ranges that start on odd tiles, cross
    parents and heads, and end in the middle of a parent."""
    for seed in range(RUNS):
        assert outcome(single_shot_backward_kernel, seed, *_single_shot_case(seed)) == "ok", seed


def test_model_catches_a_stage_freed_by_one_issuer_only_and_an_unguarded_overwrite():
    """Two mutations of that protocol the model must catch: mma_done counting only one thread's commit (the producer then
    reloads Q / dO under the other thread's products) and softmax warps that do not wait for the previous tile's
    products before they overwrite P / dS."""
    one = sum(outcome(single_shot_backward_kernel, s, *_single_shot_case(s), mma_done_count=1) != "ok" for s in range(80))
    two = sum(outcome(single_shot_backward_kernel, s, *_single_shot_case(s), softmax_waits_for_products=False) != "ok" for s in range(80))
    assert one > 0 and two > 0


def test_gathered_key_major_form_has_no_hazard_or_deadlock():
    """attn_dkv_pooled_loop_tc_kernel, gathered form: units of four query tiles (pieces begin and end inside one) and a ring of four stages."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        units = [rng.randint(1, 4)] + [4] * rng.randint(0, 9) + [rng.randint(1, 4)]
        assert outcome(key_major_kernel, seed, units, stages=4) == "ok", seed


def test_one_chunk_tiles_leave_a_group_without_work():
    """A list of one chunk: in one pass two of three tiles have no job for a group, in two passes one of three; it still takes part in the exchange of
    maxima and row sums."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        assert outcome(forward_kernel, seed, rng.randint(1, 7), 1, 1 + seed % 2) == "ok", seed
        assert outcome(query_major_kernel, seed, rng.randint(1, 7), rng.choice([1, 3])) == "ok", seed


@pytest.mark.parametrize("chunks", [1, 3, 8])
def test_second_round_on_fresh_barriers_has_no_hazard_or_deadlock(chunks):
    """A CTA that marked a row walks its tiles again, in two passes, over the same shared and tensor memory; commits of the first round may
    still land on that round's own barriers."""
    for seed in range(RUNS // 2):
        assert outcome(forward_kernel, seed, random.Random(seed).randint(1, 5), chunks, 1, second_round=True) == "ok", seed


def test_model_catches_a_producer_an_epilogue_warp_and_a_reader_left_out_of_the_count():
    """Three mutations of today's protocols: a query stage that counts one of its two producers, an accumulator handed back by the first of four
    epilogue warps, row sums overwritten without waiting for the epilogue."""
    producer = sum(outcome(key_major_kernel, s, _pieces(s), full_count=1) != "ok" for s in range(60))
    warp = sum(outcome(query_major_kernel, s, 7, 1, free_count=1) != "ok" for s in range(60))
    sums = sum(outcome(forward_kernel, s, 6, 1, 1, softmax_waits_for_sums=False) != "ok" for s in range(60))
    assert producer > 0 and warp > 0 and sums > 0


def test_model_catches_a_dp_buffer_handed_back_too_early():
    """Two mutations of the hand-back of dP (dQ and dense dK/dV kernels): the first of a group's four warps to have loaded its rows gives the whole
    buffer back, and warps give it back before they have loaded.  The next but one job's product then overwrites what is being read."""
    for broken in ({"dp_count": 1}, {"dp_back_first": True}):
        bad_kv = sum(outcome(key_major_kernel, s, _pieces(s), **broken) != "ok" for s in range(60))
        bad_q = sum(outcome(query_major_kernel, s, 4, 6, **broken) != "ok" for s in range(60))
        assert bad_kv > 0 and bad_q > 0, (broken, bad_kv, bad_q)


def test_two_softmax_groups_have_no_hazard_or_deadlock():
    """attn_fwd_pooled_loop_tc_kernel as short lists get it: two groups on three S buffers, so that a group's buffer changes from job to job; one
    to four chunks, one pass and two, and a second round."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        tiles, chunks = rng.randint(1, 7), rng.randint(1, 4)
        assert outcome(forward_kernel, seed, tiles, chunks, 1 + seed % 2, groups=2) == "ok", seed
        assert outcome(forward_kernel, seed, tiles, chunks, 1, groups=2, second_round=True) == "ok", seed


def test_query_major_ring_of_seven_has_no_hazard_or_deadlock():
    """attn_dq_pooled_loop_tc_kernel with a remainder: seven ring stages, which no count of chunks or buffers divides."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        assert outcome(query_major_kernel, seed, rng.randint(1, 7), rng.randint(1, 9), stages=7) == "ok", seed


@pytest.mark.parametrize("head", [False, True])
def test_single_shot_forward_has_no_hazard_or_deadlock(head):
    """attn_fwd_pooled_tc_kernel with 64 keys a row (P in one part) and with 128 and 192; one tile, two, and more than the rings have stages."""
    for seed in range(RUNS):
        assert outcome(single_shot_forward_kernel, seed, 1 + seed % 9, head) == "ok", seed


@pytest.mark.parametrize("broken", [dict(sums_wait_for_epilogue=False), dict(products_wait_for_epilogue=False), dict(o_ring=2)])
def test_model_catches_a_single_shot_forward_that_does_not_wait_for_its_epilogue(broken):
    assert any(outcome(single_shot_forward_kernel, seed, 8, True, **broken) != "ok" for seed in range(60))


def test_coarse_selection_has_no_hazard_or_deadlock():
    """coarse_topk_tc_kernel alone and in clusters of two to eight; shares of one chunk, where a group is without work in either pass, odd and even ones,
    of unlike length."""
    for seed in range(RUNS):
        rng = random.Random(seed)
        low = rng.choice([1, 1, 2, 3, 8])
        assert outcome(coarse_selection_kernel, seed, [low + rng.randint(0, 1) for _ in range(rng.choice([1, 1, 2, 4, 8]))]) == "ok", seed


@pytest.mark.parametrize("broken", [dict(free_count=3), dict(groups_meet=False), dict(lists_wait=False)])
def test_model_catches_broken_coarse_selections(broken):
    assert any(outcome(coarse_selection_kernel, seed, [5, 4], **broken) != "ok" for seed in range(60))
