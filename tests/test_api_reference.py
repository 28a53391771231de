"""docs/make_api_reference.py: what it takes for a declaration."""
import importlib.util
import os

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_comments_inside_functions_document_nothing(tmp_path):
    spec = importlib.util.spec_from_file_location(
        "_api", os.path.join(ROOT, "p4app-switchML_b200", "docs", "make_api_reference.py"))
    api = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(api)
    header = tmp_path / "h.h"
    header.write_text("""// About the file.
namespace n {
// A class.
class C {
 public:
  // A method.
  void Method() {
    // A remark.
    int local = 0;
    for (;;) {
      // Another one.
      int inner = 1;
    }
  }
  // A method with arguments
  // on two lines.
  int Other(int a,
            int b) const;
};
// A function.
inline int F(const char* text = "{") {
  return 1;
}
}  // namespace n
""")
    head, entries = api.document(str(header))
    assert head == ["About the file."]
    assert [c[0] for c, _ in entries] == ["A class.", "A method.", "A method with arguments", "A function."]
