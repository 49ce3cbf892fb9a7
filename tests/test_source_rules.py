"""Rules that the device code has to keep and that no run can show to be broken: checked on the source text."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pylo_b200", "csrc")


def functions():
    """{name: body} of the device functions and kernels in the sources."""
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
        text = re.sub(r"__(?:launch_bounds|cluster_dims)__\([^()]*\)", "", text)
        for head in re.finditer(r"(?:__global__|__device__ __forceinline__)[^;{]*?(\w+)\s*\([^;{]*\)\s*\{", text):
            depth, at = 1, head.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[at], 0)
                at += 1
            out[head.group(1)] = text[head.end():at]
    return out


REACH = re.compile(r"\b(cluster_store|cluster_load|nf_at_rank)\(")


def barriers(body):
    """Cluster barriers that all threads pass, whatever branch they took: [(place, whether it orders memory accesses)]."""
    top = lambda at: body.count("{", 0, at) == body.count("}", 0, at)
    places = lambda text: [m.start() for m in re.finditer(re.escape(text), body) if top(m.start())]
    release, acquire = places('asm volatile("barrier.cluster.arrive.release'), places('asm volatile("barrier.cluster.wait.acquire')
    halves = [(at, False) for at in places("cluster_wait();")[len(places("cluster_arrive();")) - 1:]]
    return sorted([(at, True) for at in places("cluster_sync();")] + halves + [(w, True) for w in acquire if any(r < w for r in release)])


def test_no_cta_reaches_into_another_before_it_is_known_to_run():
    """Distributed shared memory may be accessed only once every CTA of the cluster has started (a cluster barrier), and read only
    behind one that orders the accesses before it; and no CTA leaves before a barrier behind the last access."""
    bodies = functions()
    seen = set()
    for name, body in bodies.items():
        reach = list(REACH.finditer(body))
        if name in ("cluster_store", "cluster_load", "nf_at_rank") or not reach or "cluster_rank()" not in body:
            continue
        seen.add(name)
        first, last = reach[0].start(), reach[-1].start()
        assert any(at < first for at, _ in barriers(body)), name
        assert any(at > last for at, ordered in barriers(body) if ordered), name
        for look in re.finditer(r"\bcluster_load\(", body):
            assert any(at < look.start() for at, ordered in barriers(body) if ordered), name
    assert {"k_factor_update", "k_small_front", "k_ns_cluster", "nf_gemm_body"} <= seen


def test_kernels_that_write_parameters_look_at_the_status_word():
    """After a wait that ran out the step's sums are incomplete; no kernel may write parameters, or VeLO's LSTM state, from them.  (k_adamw reads
    nothing that an earlier kernel of the step makes.)"""
    bodies = functions()
    for name in ("k_apply", "k_apply_adafac_cols", "k_apply_packed", "k_post_apply", "k_velo_lstm", "k_velo_mix", "k_velo_cell",
                 "k_velo_xmix"):
        assert "reported(" in bodies[name], name
    assert "poisoned" in bodies["k_apply_adafac_tc"]


def test_a_failed_wait_of_the_ring_ends_the_whole_cta():
    """A wait that runs out is one answer for the warp (shuffles and barriers follow) and, at the tile's end, for the CTA."""
    bodies = functions()
    assert "__all_sync(0xffffffffu, ok)" in bodies["pipe_wait"]
    sweep = bodies["k_state_moments"]
    assert sweep.index("block_reduce_store<NACC>") < sweep.index("dead = __syncthreads_or(dead)")


def test_the_cluster_chain_takes_in_its_copies_after_a_failed_wait():
    """k_ns_cluster's bulk copies land in other CTAs: after a wait that ran out every CTA stays until those of all are in, and the
    products are done.  That can be counted only if the failed warp starts nothing more."""
    body = functions()["k_ns_cluster"]
    assert body.count("ns_wait(") == 1 and "!__all_sync(0xffffffffu, ns_wait(" in body   # one answer for the warp
    for start in ("++products;", "++sent;"):   # products and copies of a warp that still waits only, all of them counted
        assert re.search(r"if \(warp == 0 && !dead\) \{\s*" + re.escape(start), body), start
    for word, start in (("nf_mma<", "++products;"), ("cp.async.bulk", "++sent;")):
        assert body.index(start) < body.index(word) and body.count(word) == 1
    for arrival in re.finditer(r"mbarrier\.arrive\.release\.cluster", body):
        assert "!dead" in body[body.rindex("if (", 0, arrival.start()):arrival.start()]
    told, stopped, gone = body.index("cluster_store(&sm.sent"), body.index("cluster_sync();"), body.rindex("cluster_sync();")
    assert told < stopped < body.index("pipe_wait(&sm.bar") < gone and stopped < body.index("pipe_wait(&sm.got") < gone
    assert max(body.rindex(word) for word in ("++products;", "++sent;", "say_free()")) < told
