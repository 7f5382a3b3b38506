"""The LLaMA-shape decoder in float64 torch arithmetic from the weights of a model (whole sequences, no cache)."""
import torch


class Reference:
    """Holds the weights of one rank's model as float64 CUDA tensors."""

    def __init__(self, m, layers, d, heads, kv_heads, ffn, vocab, eps=1e-5, theta=10000.0):
        get = lambda name, *shape: torch.from_numpy(m.weight(name)).cuda().double().reshape(*shape)  # noqa: E731
        self.heads, self.kv_heads, self.ffn, self.eps, self.theta = heads, kv_heads, ffn, eps, theta
        self.emb, self.gf, self.head = get("emb", vocab, d), get("gf", d), get("lm_head", vocab, d)
        self.layers = [{"g1": get(f"layers.{l}.g1", d), "g2": get(f"layers.{l}.g2", d), "qkv": get(f"layers.{l}.wqkv", (heads + 2 * kv_heads) * 128, d),
                        "o": get(f"layers.{l}.wo", d, heads * 128), "gu": get(f"layers.{l}.wgu", 2 * ffn, d), "down": get(f"layers.{l}.wdown", d, ffn)}
                       for l in range(layers)]

    def _norm(self, x, g):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + self.eps) * g

    def _rotate(self, x):
        """Neighbouring pairs of every head, token t by t / theta^(2i/128)."""
        at = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None] * self.theta ** (-2.0 * torch.arange(64, device="cuda", dtype=torch.float64) / 128)
        c, s = at.cos()[:, None], at.sin()[:, None]
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack((c * a - s * b, s * a + c * b), -1).flatten(-2)

    def logits(self, ids):
        """Logits of the last token of one sequence (a CUDA tensor of ids)."""
        x, T, Hq, Hkv = self.emb[ids.long()], ids.numel(), self.heads, self.kv_heads
        causal = torch.ones(T, T, device="cuda", dtype=torch.bool).tril()
        for w in self.layers:
            y = (self._norm(x, w["g1"]) @ w["qkv"].t()).view(T, Hq + 2 * Hkv, 128)
            q, k, v = self._rotate(y[:, :Hq]), self._rotate(y[:, Hq:Hq + Hkv]), y[:, Hq + Hkv:]
            k, v = (t.repeat_interleave(Hq // Hkv, 1) for t in (k, v))
            s = torch.einsum("qhd,khd->hqk", q, k) * 128 ** -0.5
            a = s.masked_fill(~causal, float("-inf")).softmax(-1)
            x = x + torch.einsum("hqk,khd->qhd", a, v).reshape(T, -1) @ w["o"].t()
            gu = self._norm(x, w["g2"]) @ w["gu"].t()
            x = x + (torch.nn.functional.silu(gu[:, :self.ffn]) * gu[:, self.ffn:]) @ w["down"].t()
        return self._norm(x[-1], self.gf) @ self.head.t()
