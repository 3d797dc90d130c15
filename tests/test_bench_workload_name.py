"""The workload that the bench names in its line is the one it chose: nothing in
main binds that name again."""
import ast
from pathlib import Path


def test_main_binds_the_workload_name_only_by_choosing_it():
    tree = ast.parse((Path(__file__).resolve().parents[1] / "bench.py").read_text())
    main = next(n for n in tree.body if isinstance(n, ast.FunctionDef) and n.name == "main")
    chosen = {id(t) for n in ast.walk(main) if isinstance(n, ast.Assign) for t in ast.walk(n)}
    again = [n.lineno for n in ast.walk(main)
             if isinstance(n, ast.Name) and isinstance(n.ctx, ast.Store) and n.id == "name" and id(n) not in chosen]
    assert again == []
