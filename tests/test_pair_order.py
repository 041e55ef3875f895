"""What passes between the two CTAs of a pair is ordered for a reader in the other one: signals release and waits acquire at the scope of the cluster, and the
copies of both CTAs complete on the barrier that the products wait for.  Read from the sources: an order that is missing cannot be provoked."""
import re

from test_launch_order import KERNELS, SOURCES, CSRC

import glob
import os


def _texts():
    headers = {os.path.basename(p): open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cuh"))}
    return {**headers, **{f: open(os.path.join(CSRC, f)).read() for f in SOURCES}}


def test_arrivals_at_another_cta_release_to_it():
    found = [(f, m.group()) for f, text in _texts().items() for m in re.finditer(r"mbarrier\.arrive[\w.:]*shared::cluster[\w.:]*", text)]
    assert found
    assert not [x for x in found if ".release.cluster" not in x[1]]


def test_every_wait_of_a_pair_is_of_cluster_scope():
    pairs = {k: body for k, body in KERNELS.items() if re.search(r"\bumma_f16_pair\b", body)}
    assert pairs
    for kernel, body in pairs.items():
        waits = re.findall(r"\bmbar_(?:try_|test_)?wait(?:_warp)?\b\s*(<\w+>)?", body)
        assert waits and set(waits) == {"<kClusterScope>"}, kernel
        assert re.findall(r"\bcluster_(\w+)\(\);", body) == ["sync_all", "stay"], kernel        # barriers and TMEM are handed over, the exit is not
        loads = set(re.findall(r"\btma_load_2d\w*\b", body))
        assert loads == {"tma_load_2d_pair"}, kernel
        signal = re.search(r"const uint32_t dst = [^;]*, bar = (\w+) \+ 8u \* s;", body)
        assert signal and re.search(r"\b%s = cluster_smem_addr\(full\(0\), 0\);" % signal.group(1), body), kernel
    wait = re.search(r"bool mbar_try_wait\(.*?\n}\n", _texts()["ptx_utils.cuh"], re.S).group()
    assert re.search(r"SCOPE == kClusterScope\).*?try_wait\.parity\.acquire\.cluster\.", wait, re.S)


def test_no_product_is_under_way_when_a_pair_gives_up():
    """After a wait that ran out, the warp that issues products waits (with a limit) for those it has issued before it goes to the exit."""
    for kernel, body in KERNELS.items():
        if not re.search(r"\bumma_f16_pair\b", body):
            continue
        last = max(m.end() for m in re.finditer(r"\bumma_f16_pair\b|umma_commit_pair\(acc_full", body))
        given_up = re.search(r"if \(!ok\) \{\s*if \(elect_one\(\)\) umma_commit_pair\((\w+), 1\);\s*mbar_drain\(\1, 0\);", body[last:])
        assert given_up, kernel
        assert re.search(r"mbar_init\(%s, 1\);" % given_up.group(1), body), kernel
