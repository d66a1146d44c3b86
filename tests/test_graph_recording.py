"""No collection of cycles while a CUDA graph is recorded."""
import contextlib
import gc
import threading

import pytest
import torch


def test_the_collector_stays_off_until_the_last_recording_has_ended(monkeypatch):
    from inference_b200.utils.graphs import recording

    monkeypatch.setattr(torch.cuda, "graph", lambda graph: contextlib.nullcontext())
    inside, leave = threading.Event(), threading.Event()

    def other():
        with recording(None):
            inside.set()
            leave.wait(10)

    assert gc.isenabled()
    with recording(None):
        thread = threading.Thread(target=other)
        thread.start()
        assert inside.wait(10) and not gc.isenabled()
    assert not gc.isenabled()           # the other thread still records
    leave.set()
    thread.join()
    assert gc.isenabled()
    with pytest.raises(RuntimeError), recording(None):
        raise RuntimeError("a kernel was refused")
    assert gc.isenabled()
    gc.disable()
    try:
        with recording(None):
            pass
        assert not gc.isenabled()       # a program that has switched it off finds it off
    finally:
        gc.enable()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["decode", "flux", "z_image"])
def test_recorded_steps_run_without_the_collector(kind, monkeypatch):
    device, seen = torch.device("cuda", 0), []

    def spy(owner, name):
        plain = getattr(owner, name)

        def watched(*a, **kw):
            if torch.cuda.is_current_stream_capturing():
                seen.append(gc.isenabled())
            return plain(*a, **kw)
        monkeypatch.setattr(owner, name, watched)

    if kind == "decode":
        from inference_b200.engine.llm_engine import EngineConfig, LlmEngine
        from inference_b200.models import ModelConfig
        from inference_b200.models.llama import LlamaGpu

        cfg = ModelConfig.from_json({"hidden_size": 256, "intermediate_size": 512, "num_hidden_layers": 1, "num_attention_heads": 2, "num_key_value_heads": 1,
                                     "head_dim": 128, "vocab_size": 256, "rope_theta": 10000.0})
        eng = LlmEngine(LlamaGpu(cfg, device=device).init_random(0), EngineConfig(max_batch=2, max_seq_len=64))
        spy(eng.runner, "_decode_body")
        seq = eng.new_sequence()
        eng.runner.prefill([seq], [[1, 2, 3]])
        eng.runner.decode([seq], [4])
    elif kind == "flux":
        from inference_b200.models.dit_flux import FluxConfig, FluxDiTGpu, make_ids, random_flux_weights

        cfg = FluxConfig(in_channels=16, vec_in_dim=32, context_in_dim=64, hidden_size=256, num_heads=2, depth=1, depth_single=1, guidance_embed=False)
        dit = FluxDiTGpu(cfg, device=device).load_state_dict(random_flux_weights(cfg, 0))
        spy(dit, "forward")
        txt_ids, img_ids = make_ids(4, 4, 8, device="cuda")
        rnd = lambda *s: torch.randn(*s, device="cuda").bfloat16()      # noqa: E731
        dit.forward_graphed(rnd(1, 16, cfg.in_channels), img_ids, rnd(1, 8, 64), txt_ids, torch.rand(1, device="cuda"), rnd(1, 32))
    else:
        from inference_b200.models.dit_zimage import ZImageConfig, ZImageDiTGpu, random_zimage_weights

        cfg = ZImageConfig(dim=384, n_layers=1, n_refiner_layers=1, n_heads=3, cap_feat_dim=64)
        dit = ZImageDiTGpu(cfg, device).load_state_dict(random_zimage_weights(cfg, seed=0))
        spy(dit, "forward")
        tokens = dit.refine_caption(torch.randn(1, 8, 64, device="cuda").bfloat16())
        dit.forward_graphed(torch.randn(1, 16, 8, 8, device="cuda").bfloat16(), torch.full((1,), 0.3, device="cuda"), tokens)
    assert seen and not any(seen) and gc.isenabled()
