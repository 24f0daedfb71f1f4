"""A tuning macro that a header reads reaches every source that includes the header:
the kernels of whole levels are built with the values of the separate ones."""
from cumetis_gb300 import autotune as A
from cumetis_gb300 import build as B


def test_header_macros_reach_all_sources():
    got = B.variant_defines(A.defines_by_source(dict(A.DEFAULTS, CM_TINY_MAX=32, CM_SERIAL_DEG=8, CM_MATCH_CHUNK=128)))
    match = ["-DCM_MATCH_CHUNK=128", "-DCM_SERIAL_DEG=8"]
    assert got == {"cm_match.cu": match, "cm_contract.cu": ["-DCM_TINY_MAX=32"],
                   "cm_levels.cu": sorted(match + ["-DCM_TINY_MAX=32"])}


def test_macros_of_one_source_stay_there():
    cfg = {n: next(c for c in cands if c != d) for n, d, cands, _ in A.PARAMS}
    got = B.variant_defines(A.defines_by_source(cfg))
    shared = {"CM_SERIAL_DEG", "CM_MATCH_CHUNK", "CM_TINY_MAX"}
    for name, _, _, src in A.PARAMS:
        where = {f for f, v in got.items() if any(d.startswith("-D%s=" % name) for d in v)}
        assert where == ({src, "cm_levels.cu"} if name in shared else {src}), name
    assert B.variant_defines({}) == {}
