"""Sources of the kernels that start before the kernel in front has ended (programmatic dependent launch): what a kernel of the step writes is read behind the wait and
through plain pointers.  A load through a __restrict__ pointer may be moved across the wait, and a read-only load of data that is still being written is undefined."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "aws-k8s-ansible-provisioner_b200" / "csrc"

# weights and tables; what the host uploads before a step; outputs that their kernels do not read
CONSTANTS = set("""w b bias conv_w conv_b vmix_lambda qk_gain table talk q_gain k_gain latent_gain gain gain_a gain_b gain_q gain_c gain1p gain_next sink w2 rate_log a_log
    dt_bias qw kw cos_sin router correction coef pq mu bigram pos_table delta_bias w_next b_next""".split())
UPLOADS = set("row_seq row_first row_end tiles block_table last_rows rows ctx".split())
OUTPUTS = set("""out q_out q_bf16 v_cache k_cache k_pages v_pages x x1 x2 x_next act idx weight gate_out slot_token pair_slot zero_buf step decay beta_out decay_out ring_store
    out_tokens next_in log tile_row0 tile_group n_tiles ssq slot_weight q_rot q_nope xq cache out_lat lb dst rows r_pages""".split())


def kernels():
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer("__global__", text):
            start = text.index("{", m.start())
            depth, end = 0, start
            while True:
                depth += (text[end] == "{") - (text[end] == "}")
                if depth == 0:
                    break
                end += 1
            signature = text[m.start():start]
            name = [n for n in re.findall(r"(\w+)\s*\(", signature) if n not in ("__launch_bounds__", "__cluster_dims__")]
            yield path.name, name[0] if name else signature, signature, text[start:end]


WAITING = [k for k in kernels() if "pdl_wait()" in k[3]]


def test_the_kernels_are_found():
    assert len(WAITING) > 80 and {"few_head_kernel", "logits_finish_kernel", "publish_tokens_kernel"} <= {k[1] for k in WAITING}


@pytest.mark.parametrize("kernel", WAITING, ids=lambda k: f"{k[0]}-{k[1][:40]}")
def test_written_data_is_read_through_plain_pointers(kernel):
    _, name, signature, body = kernel
    for const, arg in re.findall(r"(const\s+)?[\w:]+(?:\s+long)*\s*\*\s*__restrict__\s+(\w+)", signature):
        if const:
            activation = arg == "b" and "gain_b" in signature   # (there b is the second branch, with a gain of its own)
            assert arg in CONSTANTS | UPLOADS and not activation, f"{name}: {arg}"
        else:
            assert arg in OUTPUTS, f"{name}: {arg}"
            assert not re.search(rf"=\s*(?:\*reinterpret_cast<const [^>]*>\()?{arg}\s*\[", body), f"{name} reads {arg}"
    assert "__ldg" not in body, name
