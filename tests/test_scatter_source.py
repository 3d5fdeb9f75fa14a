"""The hand-over of the scatter's write-combining units, checked in the source: a
mistake here is a race that no run shows reliably.  A tuple in shared memory is
one scalar access (a vector access is several, in no stated order), and the
fill word is touched by atomics alone between the start and the end of an item
(a plain store beside atomics can be lost)."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def source():
    with open(os.path.join(ROOT, "partitioned_join_b200", "csrc", "pj_partition.cuh")) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def body(text, name):
    at = text.index(f"void {name}(")
    open_ = text.index("{", text.index(")\n{", at))
    depth = 0
    for i in range(open_, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[open_:i + 1]
    raise AssertionError(name)


def test_tuples_in_shared_memory_are_scalar_accesses():
    text = source()
    shared = re.findall(r"\b((?:ld|st)\.[a-z0-9_.:]*shared[a-z0-9_.:]*)", text)
    assert any(s.startswith("st.") for s in shared) and any(s.startswith("ld.") for s in shared)
    for s in shared:
        # (.v2.b64: two scalar accesses, a whole 8-byte tuple each)
        assert s.endswith((".b64", ".b128")) and ".v4" not in s, s
        assert ".relaxed.cta." in s, s


def test_fill_words_change_by_atomics_alone():
    put = body(source(), "wcu_put")
    assert re.search(r"unit_take\(&u\.fill\[", put) and "unit_free(u.fill + p" in put
    assert not re.search(r"u\.fill\[[^\]]*\]\s*=[^=]", put)
    assert not re.search(r"\bst\.", put)
    text = source()
    assert "atom.release.cta.shared.exch.b32" in text and "atom.acquire.cta.shared.add.u32" in text
    # every lane has read its sector before one of them frees the unit
    assert re.search(r"__syncwarp\(\);\s*uint32_t pos = 0;\s*if \(act && c == 0\) \{\s*unit_free\(", put)


def test_counts_stay_within_their_bits():
    # items of any length: a barrier every WCU_EPOCH tuples, each counted twice at most
    text = source()
    bits = int(re.search(r"WCU_COUNT = \(1u << (\d+)\) - 1u", text).group(1))
    epoch = int(re.search(r"WCU_EPOCH = 1u << (\d+)", text).group(1))
    assert epoch + 1 < bits
    for name in ("scatter_keys_kernel", "scatter_tuples_kernel"):
        at = text.index(f" {name}(")
        end = text.index("wcu_finish", at)
        assert re.search(r"WCU_EPOCH - 1u\)\) == 0\) __syncthreads\(\);", text[at:end]), name
    with open(os.path.join(ROOT, "partitioned_join_b200", "csrc", "pj_api.cu")) as f:
        seg = int(re.search(r"SEG_CHUNK = 1 << (\d+)", f.read()).group(1))
    assert seg < epoch   # items of batches
