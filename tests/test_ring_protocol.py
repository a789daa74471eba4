"""CPU tier: a model of the kernels' buffer ring (host logic only, no GPU code is exercised).

The tensor-core kernels hand 64-deep buffers from producer warps to the MMA thread through mbarriers that only
expose the PARITY of their phase.  Producer warp w owns the steps g with g % P == w and, before refilling buffer
g % S, waits until the buffer's "empty" barrier has completed (g // S) phases - which it can only test modulo 2.
The library therefore lets at most min(P, S) warps produce (``n_prod`` in csrc/conv_tc_hybrid.cu and
csrc/conv_tc_pair.cu).  This model replays random interleavings and checks the two facts behind that rule:
with P <= S no interleaving lets a producer overwrite a buffer the consumer has not read, and with P > S some
interleaving does."""
import random


def run(P, S, steps, seed, max_events=200000):
    """Returns True if some producer refilled a buffer that still held an unconsumed step."""
    rng = random.Random(seed)
    empty_phases = [0] * S          # completed phases of each buffer's "empty" barrier (one per consumed step)
    holds = [None] * S              # step currently stored in the buffer, None once consumed
    filled = set()                  # steps whose data has landed
    next_step = list(range(P))      # next step of each producer warp
    consumed = 0
    for _ in range(max_events):
        if consumed == steps:
            return False
        actors = [("p", w) for w in range(P) if next_step[w] < steps] + [("c", 0)]
        kind, w = rng.choice(actors)
        if kind == "p":
            g = next_step[w]
            b, use = g % S, g // S
            # parity wait: passes when the number of completed phases has the parity of `use`
            if empty_phases[b] % 2 != use % 2:
                continue
            if holds[b] is not None:
                return True         # the buffer still holds a step the consumer has not read
            holds[b] = g
            filled.add(g)
            next_step[w] += P
        else:
            g = consumed
            if g in filled and holds[g % S] == g:
                holds[g % S] = None
                empty_phases[g % S] += 1
                consumed += 1
    return False


def test_no_overwrite_when_producers_do_not_outnumber_buffers():
    for P, S in [(1, 2), (2, 2), (4, 4), (4, 5), (4, 8), (3, 3), (2, 6)]:
        for seed in range(60):
            assert not run(P, S, steps=40, seed=seed), (P, S, seed)


def test_overwrite_is_possible_with_more_producers_than_buffers():
    for P, S in [(4, 2), (4, 3), (6, 5), (8, 5)]:
        assert any(run(P, S, steps=40, seed=seed) for seed in range(400)), (P, S)


def test_ctas_that_share_a_tile_store_nothing_once_a_wait_gave_up():
    """The K split's finish (conv_tc_hybrid.cu): no wait can be made to run out here without breaking the kernel, so this
    reads the order of its steps - every CTA tells its abort to the cluster in front of the barrier, and parks and stores
    sums only if none had one to tell."""
    import os
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eccv26_tad_b200", "csrc", "conv_tc_hybrid.cu")
    text = open(path).read()
    finish = text[text.index("cluster_barrier();") - 600:text.index("// wgrad\n")]
    finish = finish[finish.index("if constexpr (SPLIT) {"):]
    told, barrier = finish.index("if (tid < G && *s_abort) store_to_cta("), finish.index("cluster_barrier();")
    known, parks = finish.index("const bool whole = *s_abort == 0;"), finish.index("if (whole && warp > FW_A_WARPS)")
    stores = finish.index("const int rows = !whole ? 0 :")
    assert finish.index("__syncthreads();") < told < barrier < known < parks < stores


def _source(name):
    import os
    return open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "eccv26_tad_b200", "csrc", name)).read()


def test_warps_that_list_pairs_meet_at_every_segment_whoever_gave_up():
    """The fp32 weight gradient's producers (conv_f32_tc.cu) list each segment's pairs between two barriers of all eight warps,
    which have no limit: a warp whose wait gave up may not miss one.  Reads the order of the steps."""
    text = _source("conv_f32_tc.cu")
    lists = text[text.index("__device__ __forceinline__ void t3_list_pairs("):]
    lists = lists[:lists.index("\n}\n")]
    assert lists.count("named_bar_sync(1, T3_A_WARPS * 32);") == 2
    assert not any(leaves in lists for leaves in ("break", "continue", "return"))
    loop = text[text.index("// one more round, which carries nothing: the end") - 3000:text.index("// one more round, which carries nothing: the end")]
    loop = loop[loop.index("for (long seg = i_begin;"):]
    assert "alive" not in loop[:loop.index("t3_list_pairs(")]
    assert loop.index("t3_list_pairs(") < loop.index("if (!alive) continue;") < loop.index("mbar_wait_warp(")


def test_no_warp_wide_step_behind_a_wait_of_single_lanes():
    """A warp in which one lane's wait gave up and another's came through never meets again.  So every wait of the tensor-core
    kernels is one lane's (its outcome shuffled, or the lane on its own from there), the whole warp's, or one whose outcome
    ``ok`` all lanes carry to the vote behind the step."""
    import re
    for name in ("conv_f32_tc.cu", "conv_tc_hybrid.cu", "conv_tc_pair.cu", "conv_tc_pairs.cu"):
        lines = _source(name).split("\n")
        for at, line in enumerate(lines):
            where = f"{name}:{at + 1}: {line.strip()}"
            if not re.search(r"\bmbar_wait\(", line) or "lane == 0" in line:
                continue
            if "bool ok = " in lines[at - 1] + line:
                rest = "\n".join(lines[at + 1:at + 50])
                to_vote = rest[:rest.index("__all_sync(0xffffffffu, ok")]
                assert "break" not in to_vote and "return" not in to_vote, where
                continue
            depth = len(line) - len(line.lstrip())
            guard = [b for b in lines[:at] if b.rstrip().endswith("{") and len(b) - len(b.lstrip()) < depth and "lane == 0" in b]
            assert guard and "elect" not in "".join(lines[at:at + 12]), where


def test_nothing_is_in_flight_when_a_cta_that_gave_up_leaves():
    """Every tensor-core kernel gives what is in flight time to finish behind a wait that gave up, before it frees tensor memory."""
    for name, kernels in (("conv_f32_tc.cu", 2), ("conv_tc_hybrid.cu", 2), ("conv_tc_pair.cu", 1), ("conv_tc_pairs.cu", 1)):
        ends = _source(name).split("tmem_dealloc")
        ends = [e for e in ends[:-1] if "tcgen05.dealloc" not in e[-200:] and "SVTAD_TABLE_ASYMMETRIC" not in e[-300:] and "void " not in e[-10:]]
        assert len(ends) == kernels and all("settle_after_abort(s_abort);" in e[-300:] for e in ends), name


def test_the_exchange_s_error_codes_are_its_own():
    """71 and 72 are documented as the exchange's; 81 to 90 as the fp32 kernels', 41 to 64 as the 16-bit ones'."""
    import re
    for name, low, high in (("conv_f32_tc.cu", 81, 90), ("conv_tc_hybrid.cu", 41, 64), ("conv_tc_pair.cu", 41, 64),
                            ("conv_tc_pairs.cu", 41, 64), ("allreduce.cu", 71, 72)):
        codes = {int(c) for c in re.findall(r", err, (\d+)\b", _source(name))}
        assert codes and low <= min(codes) and max(codes) <= high, (name, codes)
