")
                if i>=0:
                    body=cmd[i+len("open(R+'combine.cuh','w').write('''"):]; body=body[:body.index("