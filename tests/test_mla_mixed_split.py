"""Which steps give their leading single-token rows and their prompt rows different attention forms (host rule)."""
import types

from jittorinfer_b200 import ops
from jittorinfer_b200.ops import native


def meta(q, s):
    return {"q_lens": q, "s_lens": s, "total_kv": sum(s), "n_q_tiles": sum((n + 127) // 128 for n in q),
            "kv_decode": sum(x for n, x in zip(q, s) if n <= 1)}


def test_rule(monkeypatch):
    monkeypatch.setattr(ops, "_native", types.SimpleNamespace(mha_prefill_ok=native.mha_prefill_ok))
    split = lambda q, s, window=0: ops.mla_mixed_split(sum(q), 128, 64, 128, 512, 64, meta(q, s), window)      # noqa: E731
    lead, rest = split([1, 1, 1024, 1022], [1025, 1025, 1024, 1022])
    assert lead == 2 and rest["total_kv"] == 2046 and rest["n_q_tiles"] == 16 and rest["q_lens"] == [1024, 1022] and rest["kv_decode"] == 0
    assert split([1, 1], [900, 900]) is None                                   # no prompt
    assert split([1024, 1], [1024, 9000]) is None                              # no leading single tokens
    assert split([1, 40], [9000, 40]) is None                                  # the prompt is below the size that pays
    assert split([1, 100, 1], [900, 100, 5000]) is None                        # what follows is mostly a decoding context
    assert split([1, 100, 1], [900, 100, 50])[0] == 1
    assert split([1, 200], [9000, 7000], 300)[1]["s_lens"] == [7000]
    assert ops.mla_mixed_split(200, 128, 64, 128, 512, 64, None) is None and ops.mla_mixed_split(200, 128, 64, 128, 512, 64, {"total_kv": 3}) is None
