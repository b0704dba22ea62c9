"""Whole sequences of library calls recorded into a CUDA graph: the kernels that are launched as dependents of one another
(quantiser, MoE plan, row movement, GEMMs, paged metadata) replay to the bits of the eager calls on new inputs, and
DG_PDL=0 takes the programmatic edges out of the recording.  The switch is read once per process, so that
half of the check runs in processes of its own: `python test_gpu_capture.py` prints the number of those edges."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
if __name__ == "__main__":
    sys.path[:0] = [os.path.dirname(HERE), os.path.join(os.path.dirname(HERE), "deepgemm-rs_b200"), HERE]

import torch

from deepgemm import (Dtype, Operand, Output, SfGran, SfTensor, gemm_nt, moe, mqa_logits_paged, poll_device_status, quant_mx,
                      swiglu_quant, synth)

pytestmark = pytest.mark.gpu


class Steps:
    """Fixed buffers, the call sequence on them, and fresh inputs for the same buffers."""

    def __init__(self):
        dev = torch.device("cuda", 0)
        self.gen = torch.Generator(device=dev).manual_seed(1)
        self.w = {}
        for name, kind, gran, n, k in (("small", Dtype.Fp8, 128, 512, 8192), ("per32", Dtype.Fp8, 32, 512, 512), ("fp4", Dtype.Fp4, 32, 512, 512)):
            codes, sf = quant_mx(torch.randn(n, k, device=dev, generator=self.gen), n, k, kind, gran)
            self.w[name] = Operand.k_major(kind, n, k, k, sf, codes)
        self.x_small, self.x = torch.empty(16, 8192, device=dev), torch.empty(300, 512, device=dev)
        self.layer = moe.GroupedMoEFfn(synth.random_expert_weights(8, 1024, 512, 3, dev), synth.random_expert_weights(8, 512, 512, 4, dev), 8)
        self.idx, self.tw = synth.random_topk_routing(300, 8, 2, 5, dev)
        # paged indexer: 6 requests x 2 tokens, pages of 64
        self.reqs, self.per, self.heads = 6, 5, 64
        t = 2 * self.reqs
        self.q_in = torch.empty(t * self.heads, 128, device=dev)
        self.kv, kv_sf = quant_mx(torch.randn(self.reqs * self.per * 64, 128, device=dev, generator=self.gen), self.reqs * self.per * 64, 128, Dtype.Fp8, 32)
        self.kv_words = kv_sf.buf[0, :self.reqs * self.per * 64].contiguous()
        self.table = torch.randperm(self.reqs * self.per, device=dev, generator=self.gen).to(torch.int32).view(self.reqs, self.per).repeat_interleave(2, 0).contiguous()
        self.req = torch.arange(self.reqs, device=dev, dtype=torch.int32).repeat_interleave(2)
        self.lens = torch.empty(t, dtype=torch.int32, device=dev)
        self.hw = torch.randn(t, self.heads, device=dev, generator=self.gen).to(torch.bfloat16)
        self.fresh()

    def fresh(self):
        for x in (self.x_small, self.x, self.q_in):
            x.normal_(generator=self.gen)
        last = torch.randint(2, 64 * self.per + 1, (self.reqs,), device="cuda", generator=self.gen).to(torch.int32)
        self.lens.copy_(torch.stack([last - 1, last], 1).reshape(-1))

    def linear(self, x, w, gran):
        m, k = x.shape
        codes, sf = quant_mx(x, m, k, w.dtype, gran)
        y = torch.empty(m, w.rows, dtype=torch.bfloat16, device="cuda")
        gemm_nt(Operand.k_major(w.dtype, m, k, k, sf, codes), w, Output(Dtype.Bf16, m, w.rows, w.rows, y))
        return y

    def run(self):
        outs = [self.linear(self.x_small, self.w["small"], 128), self.linear(self.x, self.w["per32"], 32), self.linear(self.x, self.w["fp4"], 32)]
        codes, sf = quant_mx(self.x, 300, 512, Dtype.Fp8, 128)
        outs.append(self.layer.forward(codes, sf, self.idx, self.tw))
        h, h_sf = swiglu_quant(outs[-1], 300, 256, 128)
        t = 2 * self.reqs
        qc, qs = quant_mx(self.q_in, t * self.heads, 128, Dtype.Fp8, 32)
        logits = torch.zeros(t, 64 * self.per, dtype=torch.bfloat16, device="cuda")
        mqa_logits_paged(Operand.k_major(Dtype.Fp8, t * self.heads, 128, 128, qs, qc), self.kv, self.kv_words, self.hw, 64, self.reqs * self.per,
                         self.lens, self.req, self.table, self.per, t, self.heads, 128, logits, 64 * self.per)
        return outs + [h, h_sf.buf, logits]

    def record(self):
        self.run()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            outs = self.run()
        graph.instantiate()
        return graph, outs


def _programmatic_edges(graph):
    from cuda.bindings import runtime as rt
    g = rt.cudaGraph_t(init_value=graph.raw_cuda_graph())
    err, *_, n = rt.cudaGraphGetEdges_v2(g)
    assert err == rt.cudaError_t.cudaSuccess
    err, _, _, data, n = rt.cudaGraphGetEdges_v2(g, n)
    assert err == rt.cudaError_t.cudaSuccess
    return sum(int(d.type) == int(rt.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic) for d in data[:n])


def test_recorded_sequences_replay_on_new_inputs():
    steps = Steps()
    graph, outs = steps.record()
    assert _programmatic_edges(graph) >= 8
    for _ in range(3):
        steps.fresh()
        graph.replay()
        replayed = [o.clone() for o in outs]
        eager = steps.run()
        torch.cuda.synchronize()
        for i, (a, b) in enumerate(zip(replayed, eager)):
            assert torch.equal(a, b), f"output {i}"
    poll_device_status()


@pytest.mark.parametrize("value", ["0", "1"])
def test_switch_for_dependent_launches(value):
    out = subprocess.run([sys.executable, os.path.abspath(__file__)], env={**os.environ, "DG_PDL": value}, capture_output=True, text=True,
                         timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    edges = int(out.stdout.split()[-1])
    assert edges == 0 if value == "0" else edges >= 8


if __name__ == "__main__":
    print(_programmatic_edges(Steps().record()[0]))
