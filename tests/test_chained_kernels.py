"""Kernels that are placed before the one ahead of them ends (dep_enter) may take the read-only load
path for constant tables alone: data that path reads must not change while the kernel is resident,
and what the kernel ahead writes does."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "meumapps_ss_b200", "csrc")
TABLES = {"tw", "post", "Kp", "ops"}  # twiddles, split factors, deck constants, reduction codes


def _kernels():
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        with open(os.path.join(CSRC, name)) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        for part in src.split("__global__")[1:]:
            m = re.search(r"(k_\w+)\s*\(", part)
            if m is None:
                continue
            # the parameter list: up to the parenthesis that closes the kernel's own
            depth, i = 1, m.end()
            while depth:
                depth += {"(": 1, ")": -1}.get(part[i], 0)
                i += 1
            yield name, m.group(1), part[m.end():i - 1], part[i:]


def test_chained_kernels_read_only_tables_through_the_read_only_path():
    chained = {}
    for name, kernel, params, body in _kernels():
        if "dep_enter()" not in body:
            continue
        pars = [q.strip() for q in re.split(r",(?![^<]*>)", params)]
        chained[kernel] = [re.sub(r"\W", "", q.split()[-1]) for q in pars if "__restrict__" in q and "const" in q]
    assert {"k_stats", "k_finalize", "k_el_rows", "k_el_z", "k_axis_c", "k_axis_x", "k_z_div", "k_cols_s",
            "k_rows_r2c_s", "k_rows_c2r_s", "k_el_zsum"} <= set(chained)
    bad = {k: sorted(set(v) - TABLES) for k, v in chained.items() if set(v) - TABLES}
    assert not bad, bad
