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
    assert {n for n, relaxed in arrivals() if not relaxed} >= {"kv_full", "item_full"}


def test_issuer_waits_with_cluster_scope_where_the_other_cta_arrives():
    issuer = RAW[RAW.index("MMA issuer of the pair"):RAW.index("scheduler (CTA 0)")]
    waits = re.findall(r"!(\w+)\(&?c->(\w+)", issuer)
    assert {n for _, n in waits} == {n for n, _ in arrivals()} - {"item_full"}
    assert {f for f, _ in waits} == {"pr_wait"}


def test_every_commit_is_awaited_in_both_ctas_before_they_leave():
    committed = set(re.findall(r"umma_commit_pair\(&?c->(\w+)", CODE))
    drain = CODE[CODE.index("auto drain_mma"):CODE.index("int fail = 0;")]
    awaited = set(re.findall(r"mbar_wait(?:_abortable)?\(&?c->(\w+)", drain))
    # (the softmax warps wait for every s_full: their row sums need each sub-block's scores)
    assert committed - {"s_full"} == awaited
    # called by the issuer of CTA 0 and by the relay of CTA 1, the last commit being the one of every MMA
    assert len(re.findall(r"\bdrain_mma\(", CODE)) == 2
    assert re.search(r"umma_commit_pair\(&c->mma_done\);\s*drain_mma\(", CODE)
    assert CODE.rindex("drain_mma(") < CODE.rindex("tmem_dealloc_pair(")
