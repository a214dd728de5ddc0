"""Memory order of the tree-order sampler's decisions (k_sp_run), checked on the source: a race
there shows on no particular run. A kept point's mark is stored by one lane, so it has to be a
release that follows a warp barrier - a fence before the barrier covers that lane's own drops only -
and the look at a point's own state has to follow a fence and a barrier, since the marks of the
points around it were read by other lanes. Needs no GPU."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "surface_match_gb300", "csrc")


def _kernel(name):
    text = open(os.path.join(CSRC, "kdtree.cu")).read()
    text = re.sub(r"//[^\n]*", "", text)
    at = re.search(r"\b" + name + r"\s*\(SampleArgs a\)\s*\{", text).end()
    depth, end = 1, at
    while depth:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
    return re.sub(r"\s+", " ", text[at:end])


def test_a_kept_mark_releases_every_lanes_drops():
    body = _kernel("k_sp_run")
    drops, mark = body.index("sp_drop("), body.index("st_release(&a.dec[k], 1)")
    assert drops < mark and "__syncwarp();" in body[drops:mark]
    # nothing else marks an entry as kept
    assert not re.search(r"a\.dec\[\w+\]\s*=\s*1", body)


def test_the_own_state_is_read_after_every_lanes_look():
    body = _kernel("k_sp_run")
    look, own = body.index("sp_blocker("), body.index("ld_vol(&a.dec[k]) : 0")
    assert look < own and "fence_acq_rel(); __syncwarp();" in body[look:own]
