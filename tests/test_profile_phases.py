"""Phases to which the breakdown of a training step counts the kernels of the layers."""
import pytest

from pisceslx_b200.engine.profile_step import phase_of


@pytest.mark.parametrize("phase,kernels", [
    ("attention", ["attn_fwd_kernel<128>", "attn_stats_kernel<64, true>", "attn_bwd_fused_kernel<128>", "attn_dq_finish_kernel<64>",
                   "attn_delta_kernel<64, true>", "attn_bwd_dkv_kernel<64>", "rope_vec_kernel<false, true>"]),
    ("moe routing/permute", ["gate_topk_kernel", "gate_plan_kernel", "moe_row_dots_kernel", "moe_permute_mapped_kernel<true>"]),
    ("embedding", ["embed_rank_kernel", "embed_sum_kernel", "embed_join_kernel"]),
    ("loss", ["ce_kernel"]), ("gemm", ["gemm_sm100_kernel<256>"]), ("other", ["something_else"])])
def test_phase(phase, kernels):
    assert {phase_of("void yv::" + k) for k in kernels} == {phase}
