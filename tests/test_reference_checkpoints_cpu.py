"""Checkpoints of the UNMODIFIED reference models (the files ``__graft_entry__.build()`` copies into ``baseline/_ref``) load
into this framework's models and give the same logits, and state dicts exported here load back into the reference classes —
what a user who switches frameworks with trained ``.pth`` files in hand needs."""
import importlib.util
import os

import pytest
import torch

_REF = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "baseline", "_ref")


def _ref_module(fname):
    path = os.path.join(_REF, fname)
    if not os.path.exists(path):
        pytest.skip(f"{path} is not present (created by __graft_entry__.build() where the reference tree is)")
    spec = importlib.util.spec_from_file_location("ref_" + fname.replace(".", "_").replace("-", "_"), path)
    mod = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(mod)
    return mod


def test_gptlike_reference_state_dict_both_ways():
    ref = _ref_module("ddp_gpt_wikitext2.py")
    from llm_in_practise_b200.models.gpt import GPTLike
    torch.manual_seed(0)
    theirs = ref.GPTLike(vocab_size=200, block_size=32, n_layer=2, n_head=4, d_model=64, dropout=0.1).eval()
    for p in theirs.parameters():                                   # biases and norms away from their init values
        if p.dim() == 1:
            p.data.add_(0.1 * torch.randn_like(p))
    mine = GPTLike(vocab_size=200, block_size=32, n_layer=2, n_head=4, d_model=64, dropout=0.1).eval()
    mine.load_reference_state_dict(theirs.state_dict())
    ids = torch.randint(0, 200, (3, 24))
    with torch.no_grad():
        want = theirs(ids)
        got = mine(ids)
    got = got["logits"] if isinstance(got, dict) else got
    assert torch.allclose(got.float(), want, atol=2e-4, rtol=1e-4), (got - want).abs().max()
    # and back: a state dict exported here loads strictly into the reference class
    fresh = ref.GPTLike(vocab_size=200, block_size=32, n_layer=2, n_head=4, d_model=64, dropout=0.1).eval()
    missing, unexpected = fresh.load_state_dict(mine.reference_state_dict(), strict=False)
    assert not unexpected and set(missing) <= {"head.weight"}, (missing, unexpected)      # the head is tied to tok_emb
    with torch.no_grad():
        assert torch.allclose(fresh(ids), want, atol=2e-4, rtol=1e-4)


def test_minigpt2_reference_checkpoint_loads_in_the_tester(tmp_path):
    """``minigpt_model.pth`` exactly as llm-demo/minigpt2/model.py writes it (``model_state`` of the nn.TransformerEncoder
    model, ``stoi`` / ``itos``, ``config`` = vars(config), i.e. only what the dataset set) -> ``GPTTester``: same logits."""
    ref = _ref_module("minigpt2_model.py")
    from llm_in_practise_b200.models.minigpt import Config, GPTTester, MiniGPT2
    torch.manual_seed(0)
    text = "the quick brown fox jumps over the lazy dog " * 3
    cfg = ref.Config()
    cfg.seq_len, cfg.n_layer, cfg.n_head, cfg.embed_dim = 16, 2, 2, 32          # instance attributes: they land in vars(cfg)
    ds = ref.TextDataset(text, cfg.seq_len, cfg)
    theirs = ref.MiniGPT(cfg).eval()
    for p in theirs.parameters():
        if p.dim() == 1 or p.shape[0] == 1:
            p.data.add_(0.05 * torch.randn_like(p))
    path = tmp_path / "minigpt_model.pth"
    torch.save({"model_state": theirs.state_dict(), "stoi": ds.stoi, "itos": ds.itos, "config": vars(cfg)}, str(path))
    t = GPTTester(str(path))
    assert (t.config.n_embd, t.config.embed_dim, t.config.vocab_size) == (32, 32, len(ds.stoi))
    x = torch.stack([ds[i][0] for i in range(4)])
    with torch.no_grad():
        want, got = theirs(x), t.model(x)
    assert torch.allclose(got, want, atol=2e-4, rtol=1e-4), (got - want).abs().max()
    assert t.test_output_shape() and len(t.generate("the quick", max_len=5)) == len("the quick") + 5
    # and back into the reference class
    fresh = ref.MiniGPT(cfg).eval()
    fresh.load_state_dict(t.model.reference_state_dict())
    with torch.no_grad():
        assert torch.allclose(fresh(x), want, atol=2e-4, rtol=1e-4)
    c = Config(embed_dim=48)
    assert c.n_embd == 48


def test_minigpt_reference_state_dict_loads_strictly():
    ref = _ref_module("minigpt_model.py")
    from llm_in_practise_b200.models.minigpt import MiniGPT
    torch.manual_seed(0)
    theirs = ref.MiniGPT(vocab_size=40, embed_dim=32, n_heads=2, n_layers=2, dropout=0.1).eval()
    mine = MiniGPT(40, embed_dim=32, n_heads=2, n_layers=2, dropout=0.1, reference_quirks=True).eval()
    mine.load_state_dict(theirs.state_dict(), strict=True)
    x = torch.randint(0, 40, (4, 16))
    with torch.no_grad():
        assert torch.allclose(mine(x), theirs(x), atol=1e-5)


def test_init_from_accepts_reference_and_native_files(tmp_path):
    """``PretrainConfig.init_from``: a ``.pth`` written by the reference's DDP script (module names of torch, DDP's ``module.``
    prefix, or wrapped in a checkpoint dict) and one written here both initialise the model."""
    ref = _ref_module("ddp_gpt_wikitext2.py")
    from llm_in_practise_b200.models.gpt import GPTLike
    from llm_in_practise_b200.train.pretrain import load_initial_weights
    torch.manual_seed(1)
    theirs = ref.GPTLike(vocab_size=120, block_size=16, n_layer=1, n_head=2, d_model=32, dropout=0.0).eval()
    ids = torch.randint(0, 120, (2, 12))
    with torch.no_grad():
        want = theirs(ids)
    p1, p2, p3 = (str(tmp_path / n) for n in ("final_model.pth", "ckpt.pt", "native.pth"))
    torch.save({"module." + k: v for k, v in theirs.state_dict().items()}, p1)
    torch.save({"epoch": 3, "model_state_dict": theirs.state_dict()}, p2)
    for path in (p1, p2):
        mine = GPTLike(vocab_size=120, block_size=16, n_layer=1, n_head=2, d_model=32, dropout=0.0).eval()
        assert load_initial_weights(mine, path) == "reference"
        with torch.no_grad():
            got = mine(ids)
        got = got["logits"] if isinstance(got, dict) else got
        assert torch.allclose(got, want, atol=2e-4, rtol=1e-4)
    torch.save(mine.state_dict(), p3)
    again = GPTLike(vocab_size=120, block_size=16, n_layer=1, n_head=2, d_model=32, dropout=0.0).eval()
    assert load_initial_weights(again, p3) == "native"
    with torch.no_grad():
        g2 = again(ids)
    g2 = g2["logits"] if isinstance(g2, dict) else g2
    assert torch.allclose(g2, want, atol=2e-4, rtol=1e-4)
    torch.save({"foo": torch.zeros(1)}, p3)
    with pytest.raises((ValueError, KeyError)):
        load_initial_weights(GPTLike(vocab_size=120, block_size=16, n_layer=1, n_head=2, d_model=32), p3)
