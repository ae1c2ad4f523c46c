"""Synchronisation of the D = 256 kernel on SM pairs, read from its source: a missing release or wait between the two
CTAs shows in no result until the timing is unlucky, so it is looked for here and not on a GPU."""
import re
from pathlib import Path

SOURCE = Path(__file__).resolve().parent.parent / "kernelfuser_b200" / "csrc" / "attn_fwd_pair256.cuh"
RAW = SOURCE.read_text()
CODE = re.sub(r"//[^\n]*", "", RAW)
TENSOR_MEMORY = {"p_ready", "q_ready", "o_free"}  # hand-overs of tensor memory only (tcgen05.wait and fence order those)


def arrivals():
    """(barrier, relaxed) of every arrival on a barrier of the other CTA."""
    alias = dict(re.findall(r"uint32_t (\w+) = map_to_cta\(&?c->(\w+)", CODE))
    found = re.findall(r"remote_arrive(_relaxed)?\((?:map_to_cta\(&?c->(\w+)|(\w+))", CODE)
    return [(name or alias[var], bool(relaxed)) for relaxed, name, var in found]


def test_only_tensor_memory_is_handed_over_without_a_release():
    assert {n for n, relaxed in arrivals() if relaxed} == TENSOR_MEMORY
    assert {n for n, relaxed in arrivals() if not relaxed} == {"item_full"}


def test_both_halves_of_a_stage_complete_on_the_barrier_that_the_issuer_waits_on():
    # K and V of both CTAs are read by MMAs that CTA 0 issues: a copy that completed on CTA 1's own barrier would need
    # a relay, and nothing but a release and an acquire at cluster scope would order it before the read
    assert re.search(r"full0 = map_to_cta\(c->kv_full, 0\);", CODE)
    copies = re.findall(r"(tma_load_4d\w*)\([^;]*?&tm_([kv]), ([^,]+),", CODE)
    assert sorted(c[1] for c in copies) == ["k", "v"]
    assert {(c[0], c[2]) for c in copies} == {("tma_load_4d_pair", "full0 + 8 * s")}
    assert re.findall(r"(\w*expect_tx)\(([^,]*)", CODE) == [("remote_expect_tx", "full0 + 8 * s"), ("mbar_expect_tx", "&c->q_full")]


def test_every_commit_is_awaited_in_both_ctas_before_they_leave():
    committed = set(re.findall(r"umma_commit_pair\(&?c->(\w+)", CODE))
    drain = CODE[CODE.index("auto drain_mma"):CODE.index("int fail = 0;")]
    awaited = set(re.findall(r"mbar_wait(?:_abortable)?\(&?c->(\w+)", drain))
    # (the softmax warps wait for every s_full: their row sums need each sub-block's scores)
    assert committed - {"s_full"} == awaited
    # called by the issuer of CTA 0 and by the producer of CTA 1, the last commit being the one of every MMA
    assert len(re.findall(r"\bdrain_mma\(", CODE)) == 2
    assert re.search(r"umma_commit_pair\(&c->mma_done\);\s*drain_mma\(", CODE)
    assert CODE.rindex("drain_mma(") < CODE.rindex("tmem_dealloc_pair(")
